// Inverse of one 64 x 64 complex FP32 pivot tile in shared memory by 256 threads (one CTA),
// shared by the stand-alone kernel of a slab's first tile (emg_slab.cu) and by the lookahead
// CTA of the tensor-core Gauss-Jordan update (emg_tc.cu).
//
// In-place Gauss-Jordan exchange steps with implicit pivoting, by panels of 16 columns.  Warps
// 0-3 hold panel J in registers (row r = thread / 2, eight columns per thread) and run its
// steps, one barrier of the four warps each:
//   - every warp finds its best pivot by one warp maximum over the keys (|a_rc|^2 to 17 bits,
//     63 - r) of its rows not yet used, and leaves that row and the reciprocal of its pivot
//     (formed under the maximum) in one of two shared slots;
//   - after the barrier all take the best warp's row p and exchange: every other row
//     a_r -= (a_rc / a_pc) a_p, row p times the reciprocal, column c the multipliers V_rc.
//     The columns rotate through the registers, so the loop is not unrolled over the steps.
// Meanwhile warps 4-7 apply panel J - 1 to the columns outside panels J - 1 and J as one
// rank-16 product, a_r <- [r not a pivot of the panel] a_r + sum_q V_rq a_{p_q}; all eight
// warps then apply panel J to the columns of panel J + 1.  No row is moved: with pivots
// (p_c, c) the array B holds inv[c][p_c'] = B[p_c][c'], one permutation when it is written.
//
// The tile is on the critical path of the factorization and bound by latency.  Measured a
// tile (launch included): rank-1 steps of 256 threads over the whole tile, two barriers each,
// 63 us; a panel in one warp's registers 43; this 29.
#pragma once

#include "emg_common.cuh"

namespace emg {
namespace gj {

constexpr int kTile = 64, kLd = 65, kThreads = 256, kPanel = 16, kChain = 128;

struct __align__(16) PivotShared {
    float2 row[2][kChain / 32][kPanel];    // candidate row of each warp, alternating steps
    unsigned key[2][kChain / 32];
    float2 inv[2][kChain / 32];            // the reciprocal of each warp's candidate
    int piv[kTile], ipiv[kTile], panel_of[kTile];   // pivot row of step c; its inverse; panel that used row r
    float red[kThreads / 32];
};

__device__ __forceinline__ void cmsub(float2& s, float2 a, float2 b) {   // s -= a b
    s.x = fmaf(-a.x, b.x, s.x);
    s.y = fmaf(-a.x, b.y, s.y);
    s.x = fmaf(a.y, b.y, s.x);
    s.y = fmaf(-a.y, b.x, s.y);
}
__device__ __forceinline__ void cmadd(float2& s, float2 a, float2 b) {   // s += a b
    s.x = fmaf(a.x, b.x, s.x);
    s.y = fmaf(a.x, b.y, s.y);
    s.x = fmaf(-a.y, b.y, s.x);
    s.y = fmaf(a.y, b.x, s.y);
}
// The exchange steps of panel J by threads 0..127.  used: the thread's row has been a pivot;
// changed: pivots replaced by the threshold (|pivot|^2 <= thr2, reciprocal rthr).
__device__ __forceinline__ void panel_steps(float2* Ts, int J, int tb, float thr2, float rthr, bool& used,
                                            int& changed, PivotShared& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = tid >> 1, h = tid & 1, c0 = J * kPanel;
    float2 a[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = Ts[r * kLd + c0 + 8 * h + j];
#pragma unroll 1
    for (int c = c0; c < c0 + kPanel; ++c) {
        if (c >= tb) {   // uniform: no step, only the rotation
            const float2 t = a[0];
#pragma unroll
            for (int j = 1; j < 8; ++j) a[j - 1] = a[j];
            a[7] = t;
            continue;
        }
        const int ho = (c >> 3) & 1, buf = c & 1;
        const bool owner = h == ho;
        const float m2 = fmaf(a[0].x, a[0].x, a[0].y * a[0].y);
        const unsigned key = (!owner || used) ? 0u
                                              : ((((__float_as_uint(m2) & 0x7fffffffu) >> 6) + 1u) << 6) | (unsigned)(63 - r);
        const unsigned best = __reduce_max_sync(0xffffffffu, key);
        const bool small = !(m2 > thr2);   // also catches a zero pivot
        const float s = __frcp_rn(m2);
        const float2 inv = small ? make_float2(rthr, 0.f) : make_float2(a[0].x * s, -a[0].y * s);
        float2 f;
        f.x = __shfl_sync(0xffffffffu, a[0].x, (lane & ~1) + ho);   // a_rc
        f.y = __shfl_sync(0xffffffffu, a[0].y, (lane & ~1) + ho);
        if (best && r == 63 - (int)(best & 63u)) {
            float4* slot = reinterpret_cast<float4*>(&sh.row[buf][warp][8 * h]);
#pragma unroll
            for (int j = 0; j < 4; ++j) slot[j] = make_float4(a[2 * j].x, a[2 * j].y, a[2 * j + 1].x, a[2 * j + 1].y);
            if (owner) sh.inv[buf][warp] = inv;
        }
        if (lane == 0) sh.key[buf][warp] = best;
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const uint4 ks = *reinterpret_cast<const uint4*>(&sh.key[buf][0]);
        const unsigned top = max(max(ks.x, ks.y), max(ks.z, ks.w));
        const int p = 63 - (int)(top & 63u), pw = p >> 4;
        const float2 g = sh.inv[buf][pw];
        const float4* slot = reinterpret_cast<const float4*>(&sh.row[buf][pw][8 * h]);
        float2 pr[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 v = slot[j];
            pr[2 * j] = make_float2(v.x, v.y);
            pr[2 * j + 1] = make_float2(v.z, v.w);
        }
        // the pivot row becomes the reciprocal times itself
        const bool own = r == p;
        used |= own;
        f = own ? make_float2(-g.x, -g.y) : make_float2(f.x * g.x - f.y * g.y, f.x * g.y + f.y * g.x);
        float2 last = own ? make_float2(0.f, 0.f) : a[0];
#pragma unroll
        for (int j = 1; j < 8; ++j) {
            float2 t = own ? make_float2(0.f, 0.f) : a[j];
            cmsub(t, f, pr[j]);
            a[j - 1] = t;
        }
        cmsub(last, f, pr[0]);
        a[7] = owner ? make_float2(-f.x, -f.y) : last;
        if (own && owner) {
            sh.piv[c] = p;
            sh.ipiv[p] = c;
            sh.panel_of[p] = J;
            changed += small;
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) Ts[r * kLd + c0 + 8 * h + j] = a[j];
}

// Panel J applied to one column of the threads' 16 rows r0 + i: accumulated here, stored by the
// caller once every thread has read the column's pivot rows.
template <int ROWS>
__device__ __forceinline__ void panel_apply(const float2* Ts, int J, int kq, int r0, int rs, int col, const PivotShared& sh,
                                            float2 (&acc)[ROWS]) {
#pragma unroll
    for (int i = 0; i < ROWS; ++i) acc[i] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int q = 0; q < kq; ++q) {
        const float2 b = Ts[sh.piv[J * kPanel + q] * kLd + col];
        const float2* v = Ts + r0 * kLd + J * kPanel + q;
#pragma unroll
        for (int i = 0; i < ROWS; ++i) cmadd(acc[i], v[rs * i * kLd], b);
    }
    // one rounding at the entry's magnitude, after the product
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int r = r0 + rs * i;
        if (sh.panel_of[r] == J) continue;
        const float2 x = Ts[r * kLd + col];
        acc[i] = make_float2(x.x + acc[i].x, x.y + acc[i].y);
    }
}

// Ts: 64 rows of kLd, the identity outside tb x tb (overwritten).  out (rows of ldo) and out2
// (rows of 64) receive the inverse of the tb x tb block.  Pivots of |a|^2 at or below
// rel_thr^2 max|a|^2 are replaced by that threshold and counted in *pert.  256 threads.
__device__ __forceinline__ void invert_tile(float2* Ts, int tb, float rel_thr, PivotShared& sh,
                                            int32_t* __restrict__ pert, float2* out, int64_t ldo, float2* out2) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float mx = 0.f;
#pragma unroll
    for (int i = 0; i < kTile * kTile / kThreads; ++i) {
        const int r = (tid + i * kThreads) >> 6, c = tid & 63;
        const float2 v = Ts[r * kLd + c];
        if (r < tb && c < tb) mx = fmaxf(mx, fmaf(v.x, v.x, v.y * v.y));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) sh.red[warp] = mx;
    if (tid < kTile) sh.panel_of[tid] = -1;
    __syncthreads();
    float thr2 = 0.f;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) thr2 = fmaxf(thr2, sh.red[i]);
    thr2 *= rel_thr * rel_thr;
    const float rthr = 1.f / (thr2 > 0.f ? sqrtf(thr2) : 1.f);
    bool used = (tid >> 1) >= tb;
    int changed = 0;
    const int panels = (tb + kPanel - 1) / kPanel;
#pragma unroll 1
    for (int J = 0; J < panels; ++J) {
        if (tid < kChain) {
            panel_steps(Ts, J, tb, thr2, rthr, used, changed, sh);
        } else if (J > 0) {
            // panel J - 1 on the 32 columns outside panels J - 1 and J: a column per lane, 16 rows per warp
            const int r0 = 16 * (warp - 4), blk = lane >> 4;
            const int P = blk + (blk >= J - 1) * 2;   // the blk-th of the panels 0..3 without J - 1 and J
            const int col = 16 * P + (lane & 15);
            float2 acc[16];
            panel_apply(Ts, J - 1, kPanel, r0, 1, col, sh, acc);
            asm volatile("bar.sync 2, 128;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 16; ++i) Ts[(r0 + i) * kLd + col] = acc[i];
        }
        __syncthreads();
        const int kq = min(kPanel, tb - J * kPanel);
        if (J + 1 < panels) {   // panel J on the columns of panel J + 1
            float2 acc[4];
            panel_apply(Ts, J, kq, tid >> 4, 16, 16 * (J + 1) + (tid & 15), sh, acc);
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 4; ++i) Ts[((tid >> 4) + 16 * i) * kLd + 16 * (J + 1) + (tid & 15)] = acc[i];
        } else {                // the last panel on all others
#pragma unroll 1
            for (int P = 0; P < 4; ++P) {
                if (P == J) continue;
                float2 acc[4];
                panel_apply(Ts, J, kq, tid >> 4, 16, 16 * P + (tid & 15), sh, acc);
                __syncthreads();
#pragma unroll
                for (int i = 0; i < 4; ++i) Ts[((tid >> 4) + 16 * i) * kLd + 16 * P + (tid & 15)] = acc[i];
            }
        }
        __syncthreads();
    }
    if (changed) atomicAdd(pert, changed);
#pragma unroll
    for (int i = 0; i < kTile * kTile / kThreads; ++i) {
        const int r = (tid + i * kThreads) >> 6, c = tid & 63;
        if (r < tb && c < tb) {
            const float2 x = Ts[sh.piv[r] * kLd + sh.ipiv[c]];
            out[r * ldo + c] = x;
            out2[r * kTile + c] = x;
        }
    }
}

}  // namespace gj
}  // namespace emg
