// FP64 slab factorization on the tensor cores: the rank-64 products of the block Gauss-Jordan
// inversion with FP64 results from FP16 digits, and the FP64 pivot tile on a cluster of CTAs.
//
// GB300's FP64 pipe does two FMAs per SM and clock: one 64 x 64 x 64 complex product takes
// 253 us of one SM, and a factorization spends all its time there.
//
// Products (k_prod64), from integer digit slices on a matrix unit (the scheme of Ozaki, Ogita, Oishi
// and Rump, "Error-free transformations of matrix multiplication", 2012).  Both operands are first
// scaled along K by powers of two that bring the largest entry of the tile's rows to one at every K, so
// that a badly scaled unknown costs no digits; then every operand row is scaled by the power of two
// above its largest entry and its entries are written as eight balanced radix-256 digits, 62 bits
// below that power: x = 2^E sum_i d_i 2^-(6 + 8 i), |d_0| <= 64, |d_i| <= 128.  Digits are
// exact in FP16.  The 36 digit pairs with i + j <= 7 go to eight accumulators by weight.  Over K = 64 and
// both parts of a complex operand a pair sums to at most 128 2^14 = 2^21 (half of it with one d_0), so
// accumulator s holds integers up to 2^21 max(s, 1/4) <= 7 2^21 < 2^24, exact in FP32 for every
// operand (seven radix-512 digits pass 2^24 for rows of nearly equal values).  The epilogue adds them as one
// 64-bit integer and rounds once to FP64.  What is left out, relative to the product of the scaled
// row maxima: the pairs with i + j >= 8, below 2^-52.1 at worst (2^-58 for random digits), the bits of the operands
// beyond their 62, below 2^-54, and those of the sum beyond 2^-55.  The bound is normwise: a product of
// small entries of rows with large ones keeps fewer bits than an FP64 chain of its own; normwise the product
// is closer to exact than a chain of 64 FP64 FMAs (1.0 against 3.4 half-eps for random operands, 2.0 against
// 3.8 for entries spread over six decades).  A row that holds a non-finite value gives NaN.
//
// One CTA forms a 128 (matrix columns, MMA rows) x 32 (matrix rows) tile, so that the lanes of a
// warp read and write consecutive entries of a matrix row.  Four 16-deep K chunks through two
// shared buffers (96 KB each, canonical K-major layout): all threads split the next chunk of
// both operands while the MMAs of the last run.  The 32 rows enter as N = 64, [Re | Im] for the
// real plane of the columns and [-Im | Re] for the imaginary one, so that one MMA (M = 128, N = 64,
// K = 16) serves both parts of the result: 72 per chunk, all 512 TMEM columns.  A launch of one
// wave takes 37 us, bound by the integer work of the split and the epilogue (36 with seven digits in 84
// KB, 46 with two 32-deep chunks of N = 32 MMAs one after the other); the same tiles take 250 on the FP64 pipe.
#include <algorithm>

#include "emg_gj.cuh"
#include "emg_krylov.cuh"
#include "emg_rules.cuh"

namespace emg {
namespace f64 {

constexpr int kM = 128, kN = 32, kKc = 16, kTile = 64, kThreads = 256, kDig = 8;
constexpr int kAPlane = kM * kKc * 2, kBPlane = 2 * kN * kKc * 2;   // one digit of one plane: 4 KB / 2 KB
constexpr int kBuf = 2 * kDig * (kAPlane + kBPlane);                // a chunk: 96 KB
constexpr int kSmem = 2 * kBuf;
constexpr uint32_t kTmemCols = 512;
constexpr int kNone = -(1 << 16);                                   // exponent of a zero row
constexpr unsigned long long kWaitNs = 10ull * 1000ull * 1000ull;   // bound of a wait: 10 ms
constexpr long long kSpinLimit = 1ll << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// K-major, no swizzle: K-adjacent core matrices 128 B apart, 8-row blocks 256 B apart
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) | ((uint64_t)1 << 46);
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t phase) {
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (long long it = 0; it < kSpinLimit; ++it) {
        uint32_t done = 0;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mbar), "r"(phase)
            : "memory");
        if (done) return true;
        if ((it & 63) == 63) {
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
            if (t1 - t0 > kWaitNs) return false;
            __nanosleep(256);
        }
    }
    return false;
}

__device__ __forceinline__ int expo(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }   // biased exponent

// x = t 2^(e - 1022) with |t| < 1 for biased exponents up to e (no entry is above its row's e): t 2^62 plus the bias that makes
// every digit non-negative (128 in each of the eight bytes; the sum lies between 2^62 and 2^63 + 2^63).
__device__ __forceinline__ uint64_t fixed62(double x, int e) {
    constexpr uint64_t kBias = 0x8080808080808080ull;
    const int hi = __double2hiint(x), ex = (hi >> 20) & 0x7ff;
    uint64_t m = ((uint64_t)((hi & 0xfffff) | 0x100000) << 32) | (uint32_t)__double2loint(x);
    const int sh = 9 - (e - ex);
    m = ex == 0 || sh <= -53 ? 0ull : sh >= 0 ? m << sh : m >> -sh;
    return kBias + (hi < 0 ? 0ull - m : m);
}
// digit i of two such values as a pair of FP16: byte u of 1024 + u, minus 1152
template <int I>
__device__ __forceinline__ uint32_t digit2(uint64_t a, uint64_t b) {
    constexpr uint32_t n = 3 - (I & 3), sel = n | n << 4 | (n + 4) << 8 | (n + 4) << 12;
    const uint32_t u = __byte_perm((uint32_t)(a >> (I < 4 ? 32 : 0)), (uint32_t)(b >> (I < 4 ? 32 : 0)), sel);
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"((u & 0x00ff00ffu) | 0x64006400u), "r"(0x64806480u));
    return r;
}
// the eight digits of eight K-adjacent values (K entry j relative to exponent e + sgn es[j]): one
// core-matrix row (16 bytes) per digit plane, and its negative or itself in a second place
template <bool TWO>
__device__ __forceinline__ void put_digits(const double (&v)[8], int e, const int* es, int sgn, char* dst, int plane,
                                           char* dst2, uint32_t flip) {
    uint64_t q[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) q[j] = fixed62(v[j], e + sgn * es[j]);
#define EMG_PUT(I)                                                                                                \
    {                                                                                                             \
        const uint4 x = make_uint4(digit2<I>(q[0], q[1]), digit2<I>(q[2], q[3]), digit2<I>(q[4], q[5]),            \
                                   digit2<I>(q[6], q[7]));                                                        \
        *reinterpret_cast<uint4*>(dst + (I) * plane) = x;                                                         \
        if (TWO)                                                                                                  \
            *reinterpret_cast<uint4*>(dst2 + (I) * plane) = make_uint4(x.x ^ flip, x.y ^ flip, x.z ^ flip, x.w ^ flip); \
    }
    EMG_PUT(0) EMG_PUT(1) EMG_PUT(2) EMG_PUT(3) EMG_PUT(4) EMG_PUT(5) EMG_PUT(6) EMG_PUT(7)
#undef EMG_PUT
}

// sum_s S_s 2^-(12 + 8 s) times 2^E, rounded once.  The S_s are integers, |S_s| <= 2^21 max(s, 1/4).
__device__ __forceinline__ double combine(const float (&S)[kDig], int E) {
    const int i0 = __float2int_rn(S[0]), i1 = __float2int_rn(S[1]), i2 = __float2int_rn(S[2]), i3 = __float2int_rn(S[3]);
    const int i4 = __float2int_rn(S[4]), i5 = __float2int_rn(S[5]), lo = __float2int_rn(fmaf(S[7], 0x1p-13f, S[6] * 0x1p-5f));
    long long T = (long long)(i0 * 256 + i1) << 35;   // units of 2^-55
    T += (long long)(i2 * 256 + i3) << 19;
    T += (long long)i4 * 2048 + (i5 * 8 + lo);
    unsigned long long a = T < 0 ? 0ull - (unsigned long long)T : (unsigned long long)T;
    if (a == 0 || E < -4000) return 0.0;   // (a zero row)
    const int lz = __clzll((long long)a);
    a <<= lz;
    int be = 1023 + 63 - lz + E - 55;
    a += 0x400;                                         // round at bit 11
    if (a < 0x400) { a = 1ull << 63; ++be; }            // carried out: 2^64
    if (be <= 0) return 0.0;
    const unsigned long long s = T < 0 ? 1ull << 63 : 0ull;
    if (be >= 2047) return __longlong_as_double((long long)(s | 0x7ff0000000000000ull));
    return __longlong_as_double((long long)(s | (((unsigned long long)(be - 1) << 52) + (a >> 11))));
}

// Modes of a Gauss-Jordan step k on the w x w matrix M (row-major), P = inverse of tile (k, k):
//   kRow:  rows[r][c] = sum_k P[r][k] M[k0 + k][c] for the columns outside tile k, and P itself
//          inside (rows: 64 x w); extra CTAs keep the column panel: cols[r][k] = M[r][k0 + k].
//   kRest: M[r][c] -= sum_k cols[r][k] rows[k][c] but for tile (la, la) (k_look64); columns of
//          tile k take 0 - sum (rows holds P there), rows of tile k take rows.
constexpr int kRow = 0, kRest = 1;

template <int MODE>
__global__ void __maxnreg__(200)   // 256 threads leave room on the SM for a CTA of the pivot tile's cluster
    k_prod64(int64_t w, int k, int la, double2* __restrict__ Sinv, int64_t totD, int64_t offD,
             const double2* __restrict__ pinv, double2* __restrict__ rows_, double2* __restrict__ cols_, int64_t sbuf,
             int32_t* __restrict__ status) {
    extern __shared__ __align__(1024) unsigned char dsm[];
    char* base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(dsm) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t mbar[2];
    __shared__ uint32_t tmem_base;
    __shared__ int ea[kM], eb[kN], es[kTile], bad_a[kM], bad_b[kN];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t f = blockIdx.z;
    double2* M = Sinv + f * totD + offD;
    double2* rows = rows_ + f * sbuf;
    double2* cols = cols_ + f * sbuf;
    const double2* P = pinv + f * kTile * kTile;
    const int64_t k0 = (int64_t)k * kTile, k1 = min(w, k0 + kTile);
    const int tb = (int)(k1 - k0);
    const int nct = (int)((w + kM - 1) / kM);
    const double2 z2 = make_double2(0.0, 0.0);
    int64_t c0, cend, r0, rend;        // columns and rows of the tile
    int bx = (int)blockIdx.x;
    if (MODE == kRow) {
        if (bx >= 2 * nct) {           // keep a column tile
            const int64_t q0 = (int64_t)(bx - 2 * nct) * kTile;
            for (int i = tid; i < kTile * kTile; i += kThreads) {
                const int64_t r = q0 + i / kTile;
                const int c = i % kTile;
                if (r < w) cols[r * kTile + c] = c < tb ? M[r * w + k0 + c] : z2;
            }
            return;
        }
        c0 = (int64_t)(bx >> 1) * kM;
        cend = w;
        r0 = (int64_t)(bx & 1) * kN;
        rend = tb;
        if (r0 >= rend) return;
        for (int i = tid; i < kN * kTile; i += kThreads) {   // P in the columns of tile k
            const int r = (int)r0 + i / kTile, c = i % kTile;
            if (r < tb && c < tb && k0 + c >= c0 && k0 + c < c0 + kM) rows[(int64_t)r * w + k0 + c] = P[r * kTile + c];
        }
    } else {
        c0 = (int64_t)(bx % nct) * kM;
        cend = w;
        r0 = (int64_t)(bx / nct) * kN;
        rend = w;
        if (r0 >= k0 && r0 < k1) {     // rows of tile k: the row panel (tile k is a multiple of kN rows)
            for (int i = tid; i < kN * kM; i += kThreads) {
                const int64_t r = r0 + i / kM, c = c0 + i % kM;
                if (r < k1 && c < w && (c < k0 || c >= k1)) M[r * w + c] = rows[(r - k0) * w + c];
            }
            return;
        }
        if (la >= 0 && r0 >= (int64_t)la * kTile && r0 < (int64_t)(la + 1) * kTile && c0 >= (int64_t)la * kTile &&
            min(w, c0 + kM) <= (int64_t)(la + 1) * kTile)
            return;                    // nothing but the lookahead tile
    }
    // operands: a(m, kk) = A[kk lda + m] (column c0 + m), b(n, kk) = B[n ldb + kk] (row r0 + n)
    const double2* A = MODE == kRow ? M + k0 * w + c0 : rows + c0;
    const double2* B = MODE == kRow ? P + r0 * kTile : cols + r0 * kTile;
    const int64_t lda = w;
    const int mv = (int)min((int64_t)kM, cend - c0), nv = (int)min((int64_t)kN, rend - r0);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[0])) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[1])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid < kM) { ea[tid] = kNone; bad_a[tid] = 0; }
    if (tid < kN) { eb[tid] = kNone; bad_b[tid] = 0; }
    if (tid < kTile) es[tid] = kNone;
    __syncthreads();
    // exponents: es of the tile's rows at each K, eb of row r0 + n without es, ea of column c0 + m with it
    {
        const int m = tid & (kM - 1), kh = tid >> 7;
        int xa[kTile / 2];               // all loads of both operands in flight at once
#pragma unroll
        for (int j = 0; j < kTile / 2; ++j) {
            const int q = 2 * j + kh;
            const int* p = reinterpret_cast<const int*>(A + (int64_t)q * lda + m);   // the high words
            const bool in = m < mv && q < tb;
            const int hx = in ? p[1] : 0, hy = in ? p[3] : 0;
            xa[j] = max((hx >> 20) & 0x7ff, (hy >> 20) & 0x7ff);
        }
        const int kk = tid & (kTile - 1), n0 = (tid >> 6) * (kN / 4);
        int e[kN / 4], em = kNone;
#pragma unroll
        for (int j = 0; j < kN / 4; ++j) {
            const double2 x = (n0 + j < nv && kk < tb) ? B[(int64_t)(n0 + j) * kTile + kk] : z2;
            e[j] = max(expo(x.x), expo(x.y));
            if (e[j] == 0) e[j] = kNone;
            if (e[j] == 0x7ff) bad_b[n0 + j] = 1;
            em = max(em, e[j]);
        }
        atomicMax(&es[kk], em);
        __syncthreads();
        const int s = es[kk];
#pragma unroll
        for (int j = 0; j < kN / 4; ++j) {
            const int t = __reduce_max_sync(0xffffffffu, e[j] == kNone ? kNone : e[j] - s);
            if (lane == 0) atomicMax(&eb[n0 + j], t);
        }
        int t = kNone;
#pragma unroll
        for (int j = 0; j < kTile / 2; ++j) {
            if (xa[j] == 0x7ff) bad_a[m] = 1;
            if (xa[j]) t = max(t, xa[j] + es[2 * j + kh]);
        }
        atomicMax(&ea[m], t);
    }
    // a chunk's values of this thread: column c0 + m, K block kb of 8; rows likewise, one part per thread
    const int am = tid & (kM - 1), akb = tid >> 7;
    const int bn = tid & (kN - 1), bkb = (tid >> 5) & 1, bpart = (tid >> 6) & 1;   // threads 0..127
    double2 xa[8];
    double xb[8];
    auto load = [&](int ch) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int q = ch * kKc + akb * 8 + j;
            xa[j] = (am < mv && q < tb) ? A[(int64_t)q * lda + am] : z2;
        }
        if (tid < 128) {
            const double* Bd = reinterpret_cast<const double*>(B);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int q = ch * kKc + bkb * 8 + j;
                xb[j] = (bn < nv && q < tb) ? Bd[2 * ((int64_t)bn * kTile + q) + bpart] : 0.0;
            }
        }
    };
    load(0);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t taddr = tmem_base;
    constexpr int kChunks = kTile / kKc;
    bool ok = true;
    int committed = 0;                 // chunks whose MMAs were issued (uniform)
#pragma unroll 1
    for (int ch = 0; ch < kChunks; ++ch) {
        char* abase = base + (ch & 1) * kBuf;
        char* bbase = abase + 2 * kDig * kAPlane;
        // the MMAs that read this buffer are done
        if (ch >= 2) ok = mbar_wait(smem_u32(&mbar[rules::chunk_buffer(ch - 2)]), rules::chunk_parity(ch - 2));
        {
            double v[8];
            char* dst = abase + (am >> 3) * 256 + akb * 128 + (am & 7) * 16;
            const int* e8 = es + ch * kKc + akb * 8;
            const int e = ea[am];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = xa[j].x;
            put_digits<false>(v, e, e8, -1, dst, 2 * kAPlane, nullptr, 0u);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = xa[j].y;
            put_digits<false>(v, e, e8, -1, dst + kAPlane, 2 * kAPlane, nullptr, 0u);
        }
        if (tid < 128) {
            // plane 0: rows 0-31 Re, 32-63 Im; plane 1: rows 0-31 -Im, 32-63 Re
            char* row = bbase + (bn >> 3) * 256 + bkb * 128 + (bn & 7) * 16;
            constexpr int kHalf = (kN / 8) * 256;
            if (bpart == 0)
                put_digits<true>(xb, eb[bn], es + ch * kKc + bkb * 8, 1, row, 2 * kBPlane, row + kBPlane + kHalf, 0u);
            else
                put_digits<true>(xb, eb[bn], es + ch * kKc + bkb * 8, 1, row + kHalf, 2 * kBPlane, row + kBPlane,
                                 0x80008000u);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        ok = !__syncthreads_or(!ok);           // uniform
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!ok) break;
        if (tid == 0) {
            // kind::f16: FP16 operands, FP32 accumulator, M = 128, N = 64
            constexpr uint32_t id = (1u << 4) | ((uint32_t)(2 * kN >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);
            const uint32_t a0 = smem_u32(abase), b0 = smem_u32(bbase);
#define EMG_UMMA(D, A, B, ID, ACC)                                                              \
    asm volatile(                                                                               \
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"                                       \
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(D), "l"(A), "l"(B), \
        "r"(ID), "r"(ACC)                                                                       \
        : "memory")
#pragma unroll
            for (int s = 0; s < kDig; ++s) {
                const uint32_t d = taddr + (uint32_t)(s * 2 * kN);
#pragma unroll
                for (int i = 0; i <= s; ++i) {
                    const uint64_t ad = make_desc(a0 + (uint32_t)(i * 2 * kAPlane));
                    const uint64_t bd = make_desc(b0 + (uint32_t)((s - i) * 2 * kBPlane));
                    EMG_UMMA(d, ad, bd, id, (ch == 0 && i == 0) ? 0u : 1u);
                    EMG_UMMA(d, ad + (kAPlane >> 4), bd + (kBPlane >> 4), id, 1u);
                }
            }
#undef EMG_UMMA
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&mbar[ch & 1]))
                         : "memory");
        }
        ++committed;
        if (ch + 1 < kChunks) load(ch + 1);
    }
    // this thread's outputs: column c0 + 32 (warp % 4) + lane, rows r0 + 16 (warp / 4) + n, four at a
    // time, their old values one group ahead
    const int m = (warp & 3) * 32 + lane, nb = (warp >> 2) * 16;
    const int64_t c = c0 + m;
    const bool in_k = c >= k0 && c < k1;
    double2 old[4];
    auto fetch = [&](int q) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = nb + 4 * q + j;
            old[j] = (m < mv && n < nv && !in_k) ? M[(r0 + n) * w + c] : z2;
        }
    };
    if (MODE != kRow) fetch(0);
    // the last two chunks, also after a time-out (one more bounded wait each before the TMEM goes)
    for (int c = rules::pending_from(committed); c < committed; ++c)
        if (!mbar_wait(smem_u32(&mbar[rules::chunk_buffer(c)]), rules::chunk_parity(c))) ok = false;
    ok = !__syncthreads_or(!ok);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
        const uint32_t lane_addr = taddr + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)nb;
        const int e = ea[m];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint32_t v[kDig][2][4];
#pragma unroll
            for (int s = 0; s < kDig; ++s)
#pragma unroll
                for (int p = 0; p < 2; ++p)
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(v[s][p][0]), "=r"(v[s][p][1]), "=r"(v[s][p][2]), "=r"(v[s][p][3])
                                 : "r"(lane_addr + (uint32_t)(s * 2 * kN + p * kN + 4 * q))
                                 : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            double2 cur[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) cur[j] = old[j];
            if (MODE != kRow && q < 3) fetch(q + 1);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int n = nb + 4 * q + j;
                if (m >= mv || n >= nv) continue;
                const int64_t r = r0 + n;
                float sr[kDig], si[kDig];
#pragma unroll
                for (int s = 0; s < kDig; ++s) {
                    sr[s] = __uint_as_float(v[s][0][j]);
                    si[s] = __uint_as_float(v[s][1][j]);
                }
                const int E = e + eb[n] - 2044;
                double2 x = make_double2(combine(sr, E), combine(si, E));
                if (bad_a[m] | bad_b[n]) x.x = x.y = __longlong_as_double(0x7ff8000000000000ll);
                if (MODE == kRow) {
                    if (!in_k) rows[r * w + c] = x;
                } else {
                    const bool skip = MODE == kRest && la >= 0 && r >= (int64_t)la * kTile && r < (int64_t)(la + 1) * kTile &&
                                      c >= (int64_t)la * kTile && c < (int64_t)(la + 1) * kTile;
                    if (!skip) M[r * w + c] = make_double2(cur[j].x - x.x, cur[j].y - x.y);
                }
            }
        }
    } else if (tid == 0) {
        atomicExch(status, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(kTmemCols) : "memory");
}

// The lookahead of step k on the FP64 pipe: tile (la, la) is all that the next pivot tile waits for.
//   part 0: rows[r][c] = sum_k P[r][k] M[k0 + k][c] in the columns of tile la (rows: work space)
//   part 1: M[r][c] -= sum_k M[r][k0 + k] rows[k][c] on tile (la, la)
// 128 CTAs of 8 x 4 outputs, a quarter of K per warp: 4096 cycles of an SM's FP64 pipe each.  On the
// tensor cores one 64 x 64 tile is one or two CTAs that take as long as a full wave, 35 us for
// the whole row panel before it and 33 for the tile, all on the chain of the pivot tiles; these
// two launches take 4.6 us each on the pivot tiles' stream (a 26-slab point of 311 tiles: 75 -> 55 ms
// with the row panel after them on one stream, see fp64_step's caller for both beside each other).
constexpr int kLookCtas = 128, kLookRows = 8, kLookCols = 4, kTileThreads = 128;

__device__ __forceinline__ void cmadd(double2& s, double2 a, double2 b) {   // s += a b
    s.x = fma(a.x, b.x, s.x);
    s.y = fma(a.x, b.y, s.y);
    s.x = fma(-a.y, b.y, s.x);
    s.y = fma(a.y, b.x, s.y);
}

constexpr int kPowers = 4;
struct TileWork {                      // per factor; R also holds the lookahead's row tile
    double2 X[kTile * kTile], R[kTile * kTile], P[kTile * kTile], A[kTile * kTile], Q[kTile * kTile];
    float2 seed[kTile * kTile];
    int32_t rexp[kTile];               // biased exponent of the largest entry of each row of the tile
    unsigned rmax[kPowers];            // largest |entry| of R, R^2, R^4, R^8, as float bits
    int32_t replaced;
    unsigned pad[3];                   // a multiple of 16 bytes with the above
};

// The CTA's 8 x 4 outputs of up to NA 64 x 64 x 64 products of one right operand (the second one if ``two``):
// a(r, kk, v) gives the entries of the left operands, b(kk, c) that of the right one; the sums for output
// (lane / 4, lane % 4) are returned to warp 0.
template <int NA>
struct Look {
    double2 As[NA][kLookRows][kTile + 1], Bs[kTile][kLookCols + 1], red[NA][kTileThreads / 32][32];
};
template <int NA, class FA, class FB>
__device__ __forceinline__ void look_block(Look<NA>& sm, bool two, FA a, FB b, double2 (&s)[NA]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int q = 0; q < kLookRows * kTile / kTileThreads; ++q) {
        const int i = tid + q * kTileThreads;
        double2 v[NA];
        a(i / kTile, i % kTile, v);
#pragma unroll
        for (int m = 0; m < NA; ++m)
            if (m == 0 || two) sm.As[m][i / kTile][i % kTile] = v[m];
    }
#pragma unroll
    for (int q = 0; q < kLookCols * kTile / kTileThreads; ++q) {
        const int i = tid + q * kTileThreads;
        sm.Bs[i / kLookCols][i % kLookCols] = b(i / kLookCols, i % kLookCols);
    }
    __syncthreads();
    const int r = lane / kLookCols, c = lane % kLookCols;
#pragma unroll
    for (int m = 0; m < NA; ++m) s[m] = make_double2(0.0, 0.0);
    if (NA == 1 || !two) {
#pragma unroll
        for (int kk = 0; kk < kTile / 4; ++kk) cmadd(s[0], sm.As[0][r][warp * (kTile / 4) + kk], sm.Bs[warp * (kTile / 4) + kk][c]);
    } else {
#pragma unroll
        for (int kk = 0; kk < kTile / 4; ++kk) {
            const double2 y = sm.Bs[warp * (kTile / 4) + kk][c];
#pragma unroll
            for (int m = 0; m < NA; ++m) cmadd(s[m], sm.As[m][r][warp * (kTile / 4) + kk], y);
        }
    }
#pragma unroll
    for (int m = 0; m < NA; ++m) sm.red[m][warp][lane] = s[m];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int m = 0; m < NA; ++m)
#pragma unroll
            for (int q = 1; q < kTileThreads / 32; ++q) {
                s[m].x += sm.red[m][q][lane].x;
                s[m].y += sm.red[m][q][lane].y;
            }
    }
}

__global__ void __launch_bounds__(kTileThreads) k_look64(int part, int64_t w, int k, int la, double2* Sinv, int64_t totD,
                                                         int64_t offD, const double2* pinv, TileWork* work) {
    __shared__ Look<1> sm;
    const int r0 = ((int)blockIdx.x / (kTile / kLookCols)) * kLookRows, c0 = ((int)blockIdx.x % (kTile / kLookCols)) * kLookCols;
    const int64_t f = blockIdx.z, k0 = (int64_t)k * kTile, l0 = (int64_t)la * kTile;
    double2* M = Sinv + f * totD + offD;
    double2* rows = work[f].R;
    const double2* P = pinv + f * kTile * kTile;
    const int nv = (int)min((int64_t)kTile, w - l0);   // tile k is a full one: la comes after it
    const double2 z2 = make_double2(0.0, 0.0);
    const double2* src = part == 0 ? M + k0 * w + l0 : rows;
    const int64_t ld = part == 0 ? w : kTile;
    double2 sums[1];
    look_block<1>(
        sm, false,
        [&](int r, int kk, double2 (&v)[1]) {
            v[0] = part == 0 ? P[(r0 + r) * kTile + kk] : r0 + r < nv ? M[(l0 + r0 + r) * w + k0 + kk] : z2;
        },
        [&](int kk, int c) { return c0 + c < nv ? src[(int64_t)kk * ld + c0 + c] : z2; }, sums);
    const double2 s = sums[0];
    const int r = r0 + (int)threadIdx.x / kLookCols, c = c0 + (int)threadIdx.x % kLookCols;
    if (threadIdx.x >= 32 || c >= nv) return;
    if (part == 0) {
        rows[r * kTile + c] = s;
    } else if (r < nv) {
        double2& m = M[(l0 + r) * w + l0 + c];
        m = make_double2(m.x - s.x, m.y - s.y);
    }
}

// The FP64 inverse of a pivot tile from an FP32 one.  k_seed64 inverts the tile T, scaled by a power of
// two, in FP32 (emg_gj.cuh) and rounds it to 22 bits below each column's largest entry, X.  Then T^-1 =
// X (1 + R + R^2 + ...), R = 1 - T X, in FP64, 128 CTAs a launch (k_series64).  R is formed once, and nearly
// exactly: T = T1 + T2 with the 20 bits of T1 below its rows' largest entries, so that every
// product and sum of T1 X is a multiple of one power of two and below 2^49 of it, exact in FP64, and
// the rounding of T2 X is 2^-20 of that of T X.  The series is summed by doubling, with the powers of R beside it,
//   X <- X + X R,  X <- X + X R^2,  X <- X + X R^4,  X <- X + X R^8,
// until the norm of the power (64 times its largest entry) is 3e-9 and the rest, its square, 1e-17; what is added is
// small beside X, and so is its rounding.  (Newton steps X <- X + X (1 - T X), which round 1 - T X of a final X, take
// some 25 us where this takes 31.  Against FP64 exchange steps, the error of one application with
// CUDA-core products, geometric means over 16 to 24 frequencies of two guides and two filters: theirs 1.05 to
// 1.23 times, this 0.60 to 0.87; with the products above 0.38 to 0.59 on six.)  A tile that is not near
// enough (a condition beyond some 1e5, a pivot to be replaced, values beyond FP32, NaN) is left as it was
// and k_tile64 inverts it; else that returns at once.
// A tile took 124 us in k_tile64 beside the products; the seed takes 37, a launch of the series 6 to 9.
// R^(2^i) ends the series after its launch i + 1, or is too large for it to converge soon (also a NaN)
__device__ __forceinline__ bool series_met(const TileWork& nw, int i) { return 64.f * __uint_as_float(nw.rmax[i]) <= 3e-9f; }
__device__ __forceinline__ bool series_lost(const TileWork& nw, int i) { return !(__uint_as_float(nw.rmax[i]) <= 0.1f); }

__global__ void __launch_bounds__(gj::kThreads, 1) k_seed64(int64_t w, int k, const double2* Sinv, int64_t totD, int64_t offD,
                                                            TileWork* work) {
    __shared__ float2 Ts[kTile * gj::kLd];
    __shared__ gj::PivotShared sh;
    __shared__ int s_e, rexp[kTile];
    __shared__ unsigned cmax[kTile];
    const int64_t f = blockIdx.z, k0 = (int64_t)k * kTile;
    const double2* M = Sinv + f * totD + offD + k0 * w + k0;
    TileWork& nw = work[f];
    const int tb = (int)min((int64_t)kTile, w - k0), tid = threadIdx.x;
    constexpr int kPer = kTile * kTile / gj::kThreads;
    if (tid == 0) s_e = 0;
    if (tid < kPowers) nw.rmax[tid] = 0u;
    if (tid == 0) nw.replaced = 0;
    if (tid < kTile) rexp[tid] = 0;
    if (tid < kTile) cmax[tid] = 0u;
    __syncthreads();
    double2 v[kPer];
    int e = 0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const int r = (tid + q * gj::kThreads) / kTile, c = tid % kTile;
        v[q] = (r < tb && c < tb) ? M[(int64_t)r * w + c] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int q = 0; q < kPer; ++q) {   // a warp's values are of one row
        const int r = (tid + q * gj::kThreads) / kTile;
        const int er = __reduce_max_sync(0xffffffffu, max(expo(v[q].x), expo(v[q].y)));
        if ((tid & 31) == 0) atomicMax(&rexp[r], er);
        e = max(e, er);
    }
    if ((tid & 31) == 0) atomicMax(&s_e, e);
    __syncthreads();
    // 2^-(s_e - 1023): entries below 2; out of a double's normal range k_tile64 takes the tile
    const double scale = (s_e > 0 && s_e < 2045) ? __hiloint2double((2046 - s_e) << 20, 0) : 1.0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const int r = (tid + q * gj::kThreads) / kTile, c = tid % kTile;
        Ts[r * gj::kLd + c] = (r < tb && c < tb) ? make_float2((float)(v[q].x * scale), (float)(v[q].y * scale))
                                                 : make_float2(r == c ? 1.f : 0.f, 0.f);
    }
    __syncthreads();
    gj::invert_tile(Ts, tb, 1e-6f, sh, &nw.replaced, nw.seed, kTile, nw.seed);
    if (tid < kTile) nw.rexp[tid] = tid < tb ? rexp[tid] : 1023;
    __syncthreads();
    // 22 bits below the column's largest entry: multiples of the last bit of 3 2^ec, |x| < 2^ec
    float2 x[kPer];
    unsigned top = 0u;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const int i = tid + q * gj::kThreads, r = i / kTile, c = i % kTile;
        x[q] = (r < tb && c < tb) ? nw.seed[i] : make_float2(r == c ? 1.f : 0.f, 0.f);
        top = max(top, max(__float_as_uint(x[q].x) & 0x7fffffffu, __float_as_uint(x[q].y) & 0x7fffffffu));
    }
    atomicMax(&cmax[tid % kTile], top);            // a thread's entries are of one column
    __syncthreads();
    const unsigned ec = (cmax[tid % kTile] >> 23) + 1u;   // biased; beyond FP32 the residual shows it
    const float grid = ec < 253u ? 3.f * __uint_as_float(ec << 23) : 0.f;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const int i = tid + q * gj::kThreads, r = i / kTile, c = i % kTile;
        const float xr = __fsub_rn(__fadd_rn(x[q].x, grid), grid), xi = __fsub_rn(__fadd_rn(x[q].y, grid), grid);
        const double sc = (r < tb && c < tb) ? scale : 1.0;
        nw.X[i] = make_double2(xr * sc, xi * sc);
    }
}

// Entry a of a row whose largest has biased exponent e: its bits down to 2^-20 of 2^(e - 1022) (the rest is a - this).
__device__ __forceinline__ double top_bits(double a, int e) {
    const int drop = e - expo(a) + 33;             // low bits of the 53
    const long long b = __double_as_longlong(a);
    return drop >= 53 ? 0.0 : __longlong_as_double(b & ~((1ll << drop) - 1));
}

// Launches 0 to 4 of a tile: R; X + X R and R^2; with R^2, and R^4; with R^4, and R^8; with R^8.  The one that ends the
// series stores the inverse, the later ones return at once.  A buffer is written again when its last reader is
// done: X and R; A and P; X and Q; A and R.
template <int STAGE>
__global__ void __launch_bounds__(kTileThreads) k_series64(int64_t w, int k, double2* Sinv, int64_t totD, int64_t offD,
                                                           double2* pinv, TileWork* work) {
    constexpr int NA = STAGE == 4 ? 1 : 2;
    __shared__ Look<NA> sm;
    const int r0 = ((int)blockIdx.x / (kTile / kLookCols)) * kLookRows, c0 = ((int)blockIdx.x % (kTile / kLookCols)) * kLookCols;
    const int64_t f = blockIdx.z, k0 = (int64_t)k * kTile;
    double2* T = Sinv + f * totD + offD + k0 * w + k0;
    TileWork& nw = work[f];
    const int tb = (int)min((int64_t)kTile, w - k0);
    pdl_wait();
    pdl_trigger();                       // only now: waiting CTAs take shared memory from the products
    bool last = false;
    if constexpr (STAGE > 0) {
#pragma unroll
        for (int i = 0; i < STAGE; ++i)
            if (series_lost(nw, i) || (i + 1 < STAGE && series_met(nw, i))) return;   // k_tile64's, or done
        last = series_met(nw, STAGE - 1);
        if (STAGE == kPowers && !last) return;
    }
    const double2* left = STAGE == 2 || STAGE == 4 ? nw.A : nw.X;         // the sum so far
    const double2* right = STAGE == 0 ? nw.X : STAGE == 2 ? nw.P : STAGE == 3 ? nw.Q : nw.R;   // the power of R
    double2 s[NA];
    look_block<NA>(
        sm, NA == 2 && !last,
        [&](int r, int kk, double2 (&v)[NA]) {
            r += r0;
            if constexpr (STAGE == 0) {
                const double2 a = r < tb && kk < tb ? T[(int64_t)r * w + kk] : make_double2(r == kk ? 1.0 : 0.0, 0.0);
                const int e = nw.rexp[r];
                v[0] = make_double2(top_bits(a.x, e), top_bits(a.y, e));
                v[1] = make_double2(a.x - v[0].x, a.y - v[0].y);
            } else {
                v[0] = left[r * kTile + kk];
                if constexpr (NA == 2) v[1] = last ? make_double2(0.0, 0.0) : right[r * kTile + kk];
            }
        },
        [&](int kk, int c) { return right[kk * kTile + c0 + c]; }, s);
    if (threadIdx.x >= 32) return;
    const int r = r0 + (int)threadIdx.x / kLookCols, c = c0 + (int)threadIdx.x % kLookCols, o = r * kTile + c;
    double2 p = s[NA - 1];               // the next power, or R
    if constexpr (STAGE == 0) {
        p = make_double2((r == c ? 1.0 : 0.0) - s[0].x - s[1].x, -s[0].y - s[1].y);
    } else {
        const double2 x = left[o], v = make_double2(x.x + s[0].x, x.y + s[0].y);
        if (!last) {
            (STAGE == 2 ? nw.X : nw.A)[o] = v;
        } else {
            if (r < tb && c < tb) {
                T[(int64_t)r * w + c] = v;
                pinv[(f * kTile + r) * kTile + c] = v;
            }
            return;
        }
    }
    (STAGE == 1 ? nw.P : STAGE == 2 ? nw.Q : nw.R)[o] = p;
    const double m = fmax(fabs(p.x), fabs(p.y));
    const float mf = (m <= 3e38 && p.x == p.x && p.y == p.y) ? __double2float_ru(m) : __int_as_float(0x7f800000);
    const unsigned best = __reduce_max_sync(0xffffffffu, __float_as_uint(mf));
    if (threadIdx.x == 0) atomicMax(&nw.rmax[min(STAGE, kPowers - 1)], best);
}

// FP64 inverse of pivot tile k by a cluster of 16 CTAs of 128 threads: in-place Gauss-Jordan exchange
// steps with implicit pivoting (see emg_gj.cuh for the FP32 form), four columns per CTA, thread
// (row t / 2, columns 2 (t % 2), + 1).  CTA J runs the four steps of its own panel, the others
// read the multipliers and pivot rows from its shared memory after a cluster barrier and apply
// them to their columns as a rank-4 product, so the 1 M FMAs of a tile are spread over 16 SMs'
// FP64 pipes.  Pivots compare max(|re|, |im|) (14 bits of it, the lowest row on ties); a pivot of
// |a|^2 at or below rel_thr^2 max|a|^2 is replaced by that threshold and counted.  One CTA took
// 600 us a tile (85 % of its FP64 pipe), this 115 (124 while products run beside it).  It takes the
// tiles that the series leaves.
constexpr int kRanks = 16, kPc = 4;

__device__ __forceinline__ double2 remote(const double2* p, int rank) {
    uint32_t a;
    double2 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__global__ void __launch_bounds__(kTileThreads) k_tile64(int64_t w, int k, double2* __restrict__ Sinv, int64_t totD,
                                                         int64_t offD, double2* __restrict__ pinv, double rel_thr,
                                                         int32_t* __restrict__ perturbed, const TileWork* __restrict__ work) {
    struct __align__(16) Shared {
        double2 V[kTile][kPc];                 // multipliers of this CTA's panel
        double2 row[2][kTileThreads / 32][kPc];   // candidate row of each warp
        double2 prow[kPc][kPc];                // pivot rows of the panel being applied, own columns
        double2 mx;                            // (local maximum, unused)
        int4 pivots;                           // pivot rows of this CTA's steps (-1: none)
        unsigned key[2][kTileThreads / 32];
        int piv[kTile], ipiv[kTile];
        double red[kTileThreads / 32];
    };
    __shared__ Shared sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = tid >> 1, h = tid & 1;
    const int rank = (int)blockIdx.x;
    const int64_t f = blockIdx.z, k0 = (int64_t)k * kTile;
    for (int i = 0; i < kPowers; ++i) {     // uniform over the cluster
        if (series_lost(work[f], i)) break;
        if (series_met(work[f], i)) return;   // the inverse is there
    }
    double2* M = Sinv + f * totD + offD + k0 * w + k0;
    const int tb = (int)min((int64_t)kTile, w - k0);
    double2 a[2];
    double mx = 0.0;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int c = rank * kPc + 2 * h + j;
        if (r < tb && c < tb) {
            a[j] = M[(int64_t)r * w + c];
            mx = fmax(mx, a[j].x * a[j].x + a[j].y * a[j].y);
        } else {
            a[j] = make_double2(r == c ? 1.0 : 0.0, 0.0);
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) sh.red[warp] = mx;
    __syncthreads();
    if (tid == 0) {
        for (int i = 1; i < kTileThreads / 32; ++i) mx = fmax(mx, sh.red[i]);
        sh.mx = make_double2(mx, 0.0);
    }
    cluster_sync();
    double thr2 = remote(&sh.mx, lane & (kRanks - 1)).x;
#pragma unroll
    for (int o = kRanks / 2; o; o >>= 1) thr2 = fmax(thr2, __shfl_xor_sync(0xffffffffu, thr2, o));
    thr2 *= rel_thr * rel_thr;
    bool used = r >= tb;
    int changed = 0;
    const int panels = (tb + kPc - 1) / kPc;
#pragma unroll 1
    for (int J = 0; J < panels; ++J) {
        const int steps = min(kPc, tb - J * kPc);
        if (rank == J) {   // uniform per CTA
#pragma unroll
            for (int q = 0; q < kPc; ++q) {
                if (q >= steps) break;   // uniform
                const int buf = q & 1;
                const double2 v = a[q & 1];
                const bool owner = h == q / 2;
                const unsigned mag = max((unsigned)__double2hiint(v.x) & 0x7fffffffu, (unsigned)__double2hiint(v.y) & 0x7fffffffu);
                const unsigned key = (!owner || used) ? 0u : (((mag >> 6) + 1u) << 6) | (unsigned)(63 - r);
                const unsigned best = __reduce_max_sync(0xffffffffu, key);
                double2 m;   // a_rc
                m.x = __shfl_sync(0xffffffffu, v.x, (lane & ~1) + q / 2);
                m.y = __shfl_sync(0xffffffffu, v.y, (lane & ~1) + q / 2);
                if (best && r == 63 - (int)(best & 63u)) {
                    sh.row[buf][warp][2 * h] = a[0];
                    sh.row[buf][warp][2 * h + 1] = a[1];
                }
                if (lane == 0) sh.key[buf][warp] = best;
                __syncthreads();
                const uint4 ks = *reinterpret_cast<const uint4*>(&sh.key[buf][0]);
                const unsigned top = max(max(ks.x, ks.y), max(ks.z, ks.w));
                const int p = 63 - (int)(top & 63u), pw = p >> 4;
                const double2 pr0 = sh.row[buf][pw][2 * h], pr1 = sh.row[buf][pw][2 * h + 1];
                double2 g = sh.row[buf][pw][q];
                double d = g.x * g.x + g.y * g.y;
                // !(d > thr2) on the bits, off the FP64 pipe; also a zero pivot or a NaN
                const long long db = __double_as_longlong(d);
                const bool small = db <= __double_as_longlong(thr2) || db > 0x7ff0000000000000ll;
                if (small) {
                    g = make_double2(thr2 > 0.0 ? sqrt(thr2) : 1.0, 0.0);
                    d = g.x * g.x;
                }
                // the multiplier f = a_rc / g, -1 / g in the pivot row: one part per thread of the row
                const double y = __drcp_rn(d), ix = g.x * y, iy = -g.y * y;
                const bool own = r == p;
                used |= own;
                const double mx_ = own ? -1.0 : m.x, my_ = own ? 0.0 : m.y;
                const double fp = fma(h ? my_ : mx_, ix, (h ? mx_ : -my_) * iy), fo = __shfl_xor_sync(0xffffffffu, fp, 1);
                const double2 fn = h ? make_double2(-fo, -fp) : make_double2(-fp, -fo);
                double2 b0 = own ? make_double2(0.0, 0.0) : a[0], b1 = own ? make_double2(0.0, 0.0) : a[1];
                cmadd(b0, fn, pr0);
                cmadd(b1, fn, pr1);
                a[0] = owner && (q & 1) == 0 ? fn : b0;
                a[1] = owner && (q & 1) == 1 ? fn : b1;
                if (own && owner) {
                    reinterpret_cast<int*>(&sh.pivots)[q] = p;
                    changed += small;
                }
            }
            sh.V[r][2 * h] = a[0];
            sh.V[r][2 * h + 1] = a[1];
        }
        cluster_sync();
        // the panel's pivot rows and multipliers, from CTA J
        double2 v[kPc];
        if (rank != J) {
#pragma unroll
            for (int q = 0; q < kPc; ++q) v[q] = q < steps ? remote(&sh.V[r][q], J) : make_double2(0.0, 0.0);
        }
        int p[kPc];
        {
            const double2 raw = remote(reinterpret_cast<const double2*>(&sh.pivots), J);
            p[0] = __double2loint(raw.x);
            p[1] = __double2hiint(raw.x);
            p[2] = __double2loint(raw.y);
            p[3] = __double2hiint(raw.y);
#pragma unroll
            for (int q = 0; q < kPc; ++q)
                if (q >= steps) p[q] = -1;
        }
        bool mine = false;
#pragma unroll
        for (int q = 0; q < kPc; ++q)
            if (r == p[q]) {
                mine = true;
                sh.prow[q][2 * h] = a[0];
                sh.prow[q][2 * h + 1] = a[1];
                if (h == 0) {
                    sh.piv[J * kPc + q] = r;
                    sh.ipiv[r] = J * kPc + q;
                }
            }
        used |= mine;
        __syncthreads();
        if (rank != J) {
            double2 s0 = mine ? make_double2(0.0, 0.0) : a[0], s1 = mine ? make_double2(0.0, 0.0) : a[1];
#pragma unroll
            for (int q = 0; q < kPc; ++q) {
                if (q >= steps) break;
                cmadd(s0, v[q], sh.prow[q][2 * h]);
                cmadd(s1, v[q], sh.prow[q][2 * h + 1]);
            }
            a[0] = s0;
            a[1] = s1;
        }
        __syncthreads();   // prow is rewritten by the next panel
    }
    if (changed) atomicAdd(perturbed + f, changed);
    // array entry (p_c, c') is entry (c, p_c') of the inverse
    double2* out = pinv + f * kTile * kTile;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int c = rank * kPc + 2 * h + j;
        if (r < tb && c < tb) {
            const int ro = sh.ipiv[r], co = sh.piv[c];
            M[(int64_t)ro * w + co] = a[j];
            out[ro * kTile + co] = a[j];
        }
    }
    cluster_sync();   // no CTA leaves while its shared memory is read
}

}  // namespace f64

// Launch hooks (declared in emg_krylov.cuh).
int64_t fp64_tile_work() { return sizeof(f64::TileWork); }

int fp64_tile(int64_t w, int k, int64_t F, double2* Sinv, int64_t totD, int64_t offD, double2* pinv, double rel_thr,
              int32_t* perturbed, void* work, cudaStream_t st) {
    static bool attr[64] = {false};   // per device
    int dev = 0;
    EMG_CUDA(cudaGetDevice(&dev));
    if (dev >= 64 || !attr[dev]) {
        EMG_CUDA(cudaFuncSetAttribute(f64::k_tile64, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        // they run beside k_prod64, which needs most of an SM's shared memory: another split of it would make
        // the SM drain first
        constexpr auto kCarve = cudaFuncAttributePreferredSharedMemoryCarveout;
        EMG_CUDA(cudaFuncSetAttribute(f64::k_tile64, kCarve, cudaSharedmemCarveoutMaxShared));
        EMG_CUDA(cudaFuncSetAttribute(f64::k_seed64, kCarve, cudaSharedmemCarveoutMaxShared));
        EMG_CUDA(cudaFuncSetAttribute(f64::k_series64<0>, kCarve, cudaSharedmemCarveoutMaxShared));
        EMG_CUDA(cudaFuncSetAttribute(f64::k_series64<1>, kCarve, cudaSharedmemCarveoutMaxShared));
        EMG_CUDA(cudaFuncSetAttribute(f64::k_series64<2>, kCarve, cudaSharedmemCarveoutMaxShared));
        EMG_CUDA(cudaFuncSetAttribute(f64::k_series64<3>, kCarve, cudaSharedmemCarveoutMaxShared));
        EMG_CUDA(cudaFuncSetAttribute(f64::k_series64<4>, kCarve, cudaSharedmemCarveoutMaxShared));
        EMG_CUDA(cudaFuncSetAttribute(f64::k_look64, kCarve, cudaSharedmemCarveoutMaxShared));
        if (dev < 64) attr[dev] = true;
    }
    auto* nw = static_cast<f64::TileWork*>(work);
    f64::k_seed64<<<dim3(1, 1, (unsigned)F), gj::kThreads, 0, st>>>(w, k, Sinv, totD, offD, nw);
    EMG_CUDA(cudaGetLastError());
    for (int i = 0; i < 5; ++i) {
        auto stage = i == 0   ? f64::k_series64<0>
                     : i == 1 ? f64::k_series64<1>
                     : i == 2 ? f64::k_series64<2>
                     : i == 3 ? f64::k_series64<3>
                              : f64::k_series64<4>;
        EMG_CUDA(launch_pdl(stage, dim3(f64::kLookCtas, 1, (unsigned)F), dim3(f64::kTileThreads), 0, st, 0, w, k, Sinv, totD, offD,
                            pinv, nw));
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(f64::kRanks, 1, (unsigned)F);
    cfg.blockDim = dim3(f64::kTileThreads);
    cfg.stream = st;
    cudaLaunchAttribute la[1];
    la[0].id = cudaLaunchAttributeClusterDimension;
    la[0].val.clusterDim.x = f64::kRanks;
    la[0].val.clusterDim.y = 1;
    la[0].val.clusterDim.z = 1;
    cfg.attrs = la;
    cfg.numAttrs = 1;
    EMG_CUDA(cudaLaunchKernelEx(&cfg, f64::k_tile64, w, k, Sinv, totD, offD, pinv, rel_thr, perturbed,
                                static_cast<const f64::TileWork*>(nw)));
    return EMG_OK;
}

int fp64_step(int stage, int64_t w, int k, int la, int64_t F, double2* Sinv, int64_t totD, int64_t offD, const double2* pinv,
              double2* rows, double2* cols, int64_t sbuf, void* work, int32_t* status, cudaStream_t st) {
    static bool attr[64] = {false};   // per device
    int dev = 0;
    EMG_CUDA(cudaGetDevice(&dev));
    if (dev >= 64 || !attr[dev]) {
        EMG_CUDA(cudaFuncSetAttribute(f64::k_prod64<f64::kRow>, cudaFuncAttributeMaxDynamicSharedMemorySize, f64::kSmem + 1024));
        EMG_CUDA(cudaFuncSetAttribute(f64::k_prod64<f64::kRest>, cudaFuncAttributeMaxDynamicSharedMemorySize, f64::kSmem + 1024));
        constexpr auto kCarve = cudaFuncAttributePreferredSharedMemoryCarveout;
        EMG_CUDA(cudaFuncSetAttribute(f64::k_prod64<f64::kRow>, kCarve, cudaSharedmemCarveoutMaxShared));
        EMG_CUDA(cudaFuncSetAttribute(f64::k_prod64<f64::kRest>, kCarve, cudaSharedmemCarveoutMaxShared));
        if (dev < 64) attr[dev] = true;
    }
    const unsigned nct = (unsigned)((w + f64::kM - 1) / f64::kM), nrt = (unsigned)((w + f64::kN - 1) / f64::kN);
    const unsigned nt = (unsigned)((w + f64::kTile - 1) / f64::kTile);
    constexpr int sm = f64::kSmem + 1024;
    if (stage == 0)
        for (int part = 0; part < 2; ++part)
            f64::k_look64<<<dim3(f64::kLookCtas, 1, (unsigned)F), f64::kTileThreads, 0, st>>>(part, w, k, la, Sinv, totD, offD,
                                                                                            pinv,
                                                                                            static_cast<f64::TileWork*>(work));
    else if (stage == 1)
        f64::k_prod64<f64::kRow><<<dim3(2 * nct + nt, 1, (unsigned)F), f64::kThreads, sm, st>>>(
            w, k, la, Sinv, totD, offD, pinv, rows, cols, sbuf, status);
    else
        f64::k_prod64<f64::kRest><<<dim3(nct * nrt, 1, (unsigned)F), f64::kThreads, sm, st>>>(
            w, k, la, Sinv, totD, offD, pinv, rows, cols, sbuf, status);
    EMG_CUDA(cudaGetLastError());
    return EMG_OK;
}
}  // namespace emg
