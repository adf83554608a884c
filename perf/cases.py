"""Performance cases: the framework's hot path through its public entry points.

Three families, as a user's program meets them:

* volume assembly (``AssemblyPlan.assemble`` / ``assemble_tensor``): one fill of E and B
  on jittered Kuhn boxes, from a few hundred tets to the 80^3 cube of the assembly
  micro-benchmark;
* frequency solves: forming A(k) and residuals of a sweep (``RestrictedSystem``),
  per-point direct solves (``FrequencySweep.run``), batched sweeps
  (``run_anchored``, ``run_warm``) and the drop-in solver slot (``GPUSolver.solve``)
  on the WR-90 guide and the five-cavity iris filter;
* cavity eigenmodes (``CavityEigen.solve``).

``prepare`` makes a program's state from the seed (jittered vertices, materials,
frequencies); ``run`` is one pass; ``work`` the least bytes and operations of one pass;
``exact`` the same results in plain 64-bit torch.
"""
from __future__ import annotations

import copy
import functools
import itertools
import math

import numpy as np
import torch

from emerge_gb300.assembly import AssemblyPlan
from emerge_gb300.eigen import CavityEigen, box_sigma
from emerge_gb300.freq import Assembler
from emerge_gb300.geometry import dielectric_cavity, iris_filter, straight_waveguide
from emerge_gb300.mesh import Nedelec2Basis, TetMesh, structured_box
from emerge_gb300.solver import FrequencySweep, GPUSolver

C0 = 299792458.0
BAND = {"wr90": (8.2e9, 12.4e9), "iris": (8.0e9, 12.0e9)}


def listed():
    return [
        # a toy mesh: every launch and every host step of a fill counts
        {"name": "assemble-tiny", "kind": "assemble", "nx": 4, "ny": 3, "nz": 5, "mat": "dielectric"},
        # an ordinary part mesh with lossy magnetic material (complex mu: E is complex too)
        {"name": "assemble-lossy", "kind": "assemble", "nx": 24, "ny": 31, "nz": 19, "mat": "magnetic"},
        # the assembly micro-benchmark: 80^3 cells, lossy dielectric, mu = 1
        {"name": "assemble-cube80", "kind": "assemble", "nx": 80, "ny": 80, "nz": 80, "mat": "dielectric"},
        # full (3,3) material tensors in every tet
        {"name": "assemble-tensor", "kind": "assemble", "nx": 21, "ny": 22, "nz": 23, "mat": "tensor"},
        # forming A(k) for a chunk of a sweep and checking its residuals
        {"name": "residual-sweep", "kind": "residual", "structure": "iris", "h": 4.0, "nf": 45},
        # one port-driven frequency point solved directly in FP64 (the accuracy reference of a sweep)
        {"name": "point-fp64", "kind": "points", "structure": "wr90", "h": 3.0, "nf": 1, "precond": "slab64"},
        # per-point FP32 factor with FP64 refinement on the filter of the sweep benchmark (306,832 unknowns)
        {"name": "point-fp32", "kind": "points", "structure": "iris", "h": 2.0, "nf": 1, "precond": "slab32"},
        # the batched sweep of a filter, the band in two halves with one anchor factor each
        {"name": "sweep-filter", "kind": "bands", "structure": "iris", "h": 3.0, "nf": 48},
        # the warm-started sweep: few training columns, then the rest from their span
        {"name": "sweep-warm", "kind": "warm", "structure": "wr90", "h": 2.5, "nf": 101, "train": 8},
        # a coarse guide and a few points: latency of the whole solve path
        {"name": "sweep-coarse", "kind": "bands", "structure": "wr90", "h": 6.0, "nf": 10},
        # the reference's solver slot: host CSR matrix and right-hand side in, solution out
        {"name": "solver-slot", "kind": "slot", "structure": "wr90", "h": 4.0},
        # lowest modes of a dielectric-loaded cavity
        {"name": "cavity-modes", "kind": "eigen", "a": 22.0, "b": 18.0, "c": 27.0, "h": 3.0, "modes": 6},
    ]


def draw(rng):
    """One more case of the listed families and ranges."""
    kind = rng.choice(["assemble", "assemble", "assemble", "residual", "points", "bands", "warm", "slot", "eigen"])
    if kind == "assemble":
        mat = rng.choice(["dielectric", "magnetic", "tensor"])
        top = 40 if mat == "tensor" else 80
        n = [int(round(2 * (top / 2) ** rng.random())) for _ in range(3)]
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "mat": mat}
    structure = rng.choice(["wr90", "iris"])
    h = round(rng.uniform(3.0, 6.0) if structure == "iris" else rng.uniform(2.8, 7.0), 2)
    if kind == "residual":
        return {"kind": kind, "structure": structure, "h": max(h, 4.0), "nf": rng.randint(1, 45)}
    if kind == "points":
        if rng.random() < 0.5:
            return {"kind": kind, "structure": "wr90", "h": max(h, 3.0), "nf": 1, "precond": "slab64"}
        return {"kind": kind, "structure": structure, "h": h, "nf": rng.randint(1, 2), "precond": "slab32"}
    if kind == "bands":
        return {"kind": kind, "structure": structure, "h": h, "nf": int(round(4 * 12 ** rng.random()))}
    if kind == "warm":
        return {"kind": kind, "structure": "wr90", "h": max(h, 2.8), "nf": int(round(20 * 5 ** rng.random())),
                "train": rng.randint(4, 12)}
    if kind == "slot":
        return {"kind": kind, "structure": "wr90", "h": round(rng.uniform(3.6, 7.0), 2)}
    a, b, c = (round(rng.uniform(15.0, 24.0), 1) for _ in range(3))
    return {"kind": kind, "a": a, "b": b, "c": c, "h": round(rng.uniform(3.2, 4.5), 2), "modes": rng.randint(3, 6)}


# ------------------------------------------------------------------ meshes ---
@functools.lru_cache(maxsize=1)
def _box(nx, ny, nz):
    """Topology of an nx x ny x nz Kuhn box of unit cells (host arrays)."""
    m = structured_box(*(np.arange(n + 1.0) for n in (nx, ny, nz)))
    return m, Nedelec2Basis(m)


def _jittered(case, rng):
    """The box scaled to a unit longest side, interior vertices moved by up to 0.15 cells."""
    m0, f0 = _box(case["nx"], case["ny"], case["nz"])
    top = np.array([case["nx"], case["ny"], case["nz"]], dtype=float)[:, None]
    inside = np.all((m0.nodes > 0) & (m0.nodes < top), axis=0)
    m = copy.copy(m0)
    m.nodes = (m0.nodes + np.where(inside, rng.uniform(-0.15, 0.15, m0.nodes.shape), 0.0)) / top.max()
    d = m.nodes[:, m.edges[0]] - m.nodes[:, m.edges[1]]
    m.edge_lengths = np.sqrt(np.sum(d ** 2, axis=0))
    f = copy.copy(f0)
    f.mesh = m
    return f


@functools.lru_cache(maxsize=1)
def _guide(structure, h):
    # the filter's grid is finer along the guide, as in the sweep benchmark (2 mm and 1.3 mm)
    return iris_filter(h * 1e-3, hy=0.65e-3 * h) if structure == "iris" else straight_waveguide(h * 1e-3)


@functools.lru_cache(maxsize=1)
def _cavity(a, b, c, h):
    return dielectric_cavity(a * 1e-3, b * 1e-3, c * 1e-3, 4e-3, 10.0, h * 1e-3)


def _fill(p, rng):
    """The structure filled with a slightly lossy gas (a tolerance study's draw)."""
    er = p.er * (1.0 + 0.02 * rng.random()) * (1 - 1e-4j * rng.random())
    return er, p.ur.copy()


def _freqs(case, rng):
    lo, hi = BAND[case["structure"]]
    step = (hi - lo) / case["nf"]
    return lo + step * (np.arange(case["nf"]) + 0.1 + 0.8 * rng.random())


# ----------------------------------------------------------------- prepare ---
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "assemble":
        f = _jittered(case, rng)
        nT = f.n_tets
        loss = lambda lo, hi: rng.uniform(lo, hi, nT) * (1 - 1j * rng.uniform(0.001, 0.02, nT))  # noqa: E731
        st = {"kind": kind, "mat": case["mat"], "field": f, "plan": AssemblyPlan(f)}
        if case["mat"] == "tensor":
            def tensors(lo, hi):
                t = 0.1 * (rng.standard_normal((9, nT)) + 1j * rng.standard_normal((9, nT)))
                for k in (0, 4, 8):
                    t[k] += loss(lo, hi)
                return torch.as_tensor(t, device="cuda")
            st["eps"], st["nu"] = tensors(1, 10), tensors(0.4, 1)
        else:
            mu = loss(1, 3) if case["mat"] == "magnetic" else np.ones(nT, dtype=np.complex128)
            st["eps"] = torch.as_tensor(loss(1, 10), device="cuda")
            st["nu"] = torch.as_tensor(1.0 / mu, device="cuda")
        return st
    if kind == "eigen":
        p = _cavity(case["a"], case["b"], case["c"], case["h"])
        eps = rng.uniform(8.0, 16.0)
        er = p.er.copy()
        er[[0, 1, 2], [0, 1, 2]] = np.where(p.mesh.cell_tag == 1, eps, 1.0)
        dims = np.array([case["a"], case["b"], case["c"]]) * 1e-3
        return {"kind": kind, "modes": case["modes"], "sigma": box_sigma(dims, eps), "field": p.field,
                "cavity": CavityEigen(Assembler(), p.field, er, p.ur.copy(), p.bcs)}
    p = _guide(case["structure"], case["h"])
    er, ur = _fill(p, rng)
    freqs = _freqs(case | {"nf": case.get("nf", 1)}, rng)
    if kind == "slot":
        K, _, ids, ports = Assembler().assemble_freq_matrix(p.field, er, ur, p.bcs, float(freqs[0]))
        return {"kind": kind, "K": K[ids][:, ids].tocsr(), "b": ports[1][ids], "ids": ids, "field": p.field,
                "solver": GPUSolver()}
    sw = FrequencySweep(Assembler(), p.field, er, ur, p.bcs)
    st = {"kind": kind, "sweep": sw, "freqs": freqs, "field": p.field}
    if kind == "residual":
        k0, gam, beta = _coefficients(sw, freqs)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        cols = case["nf"] * len(sw.ports)
        x = torch.randn((sw.sys.n, cols, 2), generator=gen, device="cuda", dtype=torch.float64)
        st |= {"k2": k0 ** 2, "gam": gam, "X": torch.view_as_complex(x), "b": _rhs(sw, beta),
               "cmat": torch.arange(case["nf"], dtype=torch.int32, device="cuda").repeat_interleave(len(sw.ports))}
    return st | {k: case[k] for k in ("precond", "train") if k in case}


# --------------------------------------------------------------------- run ---
def run(state):
    kind = state["kind"]
    if kind == "assemble":
        fill = state["plan"].assemble_tensor if state["mat"] == "tensor" else state["plan"].assemble
        E, B = fill(state["eps"], state["nu"])
        return {"E": E, "B": B}
    if kind == "eigen":
        r = state["cavity"].solve(state["modes"], sigma=state["sigma"], which="LR", tol=1e-10)
        return {"k0_squared": r.eigenvalues}
    if kind == "slot":
        return {"x": state["solver"].solve(state["K"], state["b"])[0]}
    sw, f = state["sweep"], state["freqs"]
    if kind == "residual":
        A = sw.sys.form(sw.E, sw.B, state["k2"], sw.P, state["gam"])
        return {"A": A, "r": sw.sys.spmv(A, state["X"], state["cmat"], state["b"])}
    if kind == "points":
        r = sw.run(f, method="plain", precond=state["precond"], tol=1e-12, restart=40, max_iter=400)
        return {"S": r.S, "x": r.solutions}
    if kind == "bands":
        half = len(f) // 2
        rs = [sw.run_anchored(g, n_anchor=1, tol=1e-12) for g in (f[:half], f[half:])]
        return {"S": np.concatenate([r.S for r in rs]), "x": [r.solutions for r in rs]}
    # warm: the sweep in two halves, each trained on its own columns
    half = len(f) // 2
    rs = [sw.run_warm(g, n_train=state["train"], tol=1e-12, solver="anchored", n_anchor=1, restart=40)
          for g in (f[:half], f[half:])]
    return {"S": np.concatenate([r.S for r in rs]), "x": [r.solutions for r in rs]}


# -------------------------------------------------------------------- work ---
@functools.lru_cache(maxsize=64)
def _counts(structure, h, a=0.0, b=0.0, c=0.0):
    """(unknowns, nonzeros, sum w^2, sum w^3) of a restricted system and its cross-section blocks."""
    p = _cavity(a, b, c, h) if structure == "cavity" else _guide(structure, h)
    ids = Assembler(device="cpu").solve_ids(p.field, p.bcs)
    dofs = _restricted_dofs(p.field, ids)
    lev = _levels(p.field, dofs, len(ids))
    w = np.bincount(lev).astype(float)
    keys = set()
    r, q = np.repeat(dofs, 20, axis=0).ravel(), np.tile(dofs, (20, 1)).ravel()
    ok = (r >= 0) & (q >= 0)
    keys = np.unique(r[ok].astype(np.int64) * len(ids) + q[ok])
    return len(ids), len(keys), float((w ** 2).sum()), float((w ** 3).sum())


def work(case):
    kind = case["kind"]
    if kind == "assemble":
        m, f = _box(case["nx"], case["ny"], case["nz"])
        cols = _entity_columns(m)
        comp = 9 if case["mat"] == "tensor" else 1
        # values of E and B once, the pattern, tet data and materials once; ~20 x 20 entries
        # of two matrices per tet at 8 operations each
        return {"bytes": 32.0 * cols + 4.0 * cols + m.n_tets * (96 + 32.0 * comp) + 24.0 * m.n_nodes,
                "flops": m.n_tets * 400 * 2 * 8.0}
    if kind == "eigen":
        n, nnz, w2, w3 = _counts("cavity", case["h"], case["a"], case["b"], case["c"])
        cols = 4.0 * case["modes"]
        return {"bytes": 16.0 * (w2 + 2 * w2 * cols / 4), "flops": 8.0 * w3 + cols * (16.0 * w2 + 16.0 * nnz)}
    n, nnz, w2, w3 = _counts(case["structure"], case["h"])
    nf = case.get("nf", 1)
    cols = 2.0 * nf
    if kind == "residual":
        return {"bytes": 16.0 * (4 * nnz + nnz * nf + 3 * n * cols), "flops": 8.0 * nnz * cols + 16.0 * nnz * nf}
    if kind == "slot":
        return {"bytes": 16.0 * (w2 + nnz), "flops": 8.0 * w3 + 16.0 * w2}
    factors = nf if kind == "points" else 2
    size = 16.0 if case.get("precond") == "slab64" else 8.0
    solved = cols if kind != "warm" else 4.0 * case["train"]
    # one block inversion per factor, one application and one product per solved column
    return {"bytes": factors * size * 3 * w2 + 16.0 * nnz * nf + 32.0 * n * cols,
            "flops": factors * 8.0 * w3 + solved * (16.0 * w2 + 8.0 * nnz)}


def _entity_columns(m):
    """Stored entries of one matrix of a Kuhn box: for every edge and face, 2 rows of twice the
    distinct edges and faces of its tets."""
    slots = np.concatenate([m.tet_to_edge, m.tet_to_tri + m.n_edges])
    if m.n_tets > 200000:     # interior average of the box: 277.4 entries per tet
        return 277.4 * m.n_tets
    n = m.n_edges + m.n_tris
    keys = np.concatenate([slots[i].astype(np.int64) * n + slots[j] for i in range(10) for j in range(10)])
    return 4 * len(np.unique(keys))


# ------------------------------------------------------------------- exact ---
def exact(case, seed):
    kind = case["kind"]
    if kind == "assemble":
        return None if case["nx"] * case["ny"] * case["nz"] > 25000 else _exact_assembly(prepare(case, seed))
    if kind == "eigen":
        return _exact_modes(prepare(case, seed))
    st = prepare(case, seed)
    if kind == "slot":
        K = st["K"].tocoo()
        lev = _levels(st["field"], _restricted_dofs(st["field"], st["ids"]), K.shape[0])
        put = lambda v: torch.as_tensor(v, device="cuda")  # noqa: E731
        x = _block_solve(put(K.row.astype(np.int64)), put(K.col.astype(np.int64)), put(K.data), lev,
                         put(st["b"])[:, None])
        return {"x": x[:, 0].cpu().numpy()}
    sw = st["sweep"]
    freqs = st["freqs"]
    k0, gam, beta = _coefficients(sw, freqs)
    row, col, at = _restricted_entries(sw)
    if kind == "residual":
        A = (sw.E[at][:, None] - torch.as_tensor(st["k2"], device="cuda") * sw.B[at][:, None]
             + torch.einsum("pk,pf->kf", sw.P[:, at], torch.as_tensor(gam, device="cuda")))
        r = st["b"].clone()
        for c, m in enumerate(st["cmat"].tolist()):
            r[:, c].index_add_(0, row, -A[:, m] * st["X"][col, c])
        return {"A": A, "r": r}
    _, nnz, w2, w3 = _counts(case["structure"], case["h"])
    if len(freqs) * (8 * w3 / 5e11 + 0.2) > 18:
        return None
    lev = _levels(st["field"], _restricted_dofs(st["field"], sw.solve_ids), sw.sys.n)
    b = _rhs(sw, beta)
    xs = []
    npo = len(sw.ports)
    for f in range(len(freqs)):
        v = sw.E[at] - k0[f] ** 2 * sw.B[at]
        for p in range(sw.P.shape[0]):
            v = v + complex(gam[p, f]) * sw.P[p, at]
        xs.append(_block_solve(row, col, v, lev, b[:, f * npo:(f + 1) * npo]))
    X = torch.cat(xs, dim=1)
    G = -(sw.u_w.T @ X).reshape(npo, len(freqs), npo).permute(1, 0, 2).cpu().numpy()    # (nf, i, j)
    P = np.asarray(sw.Pmode)
    # identical guides at both ports: the wave impedances of S_ij cancel
    S = (G - np.eye(npo)[None] * P[None, :, None]) / P[None, None, :]
    half = len(freqs) // 2 * npo
    return {"S": S, "x": X if kind == "points" else [X[:, :half], X[:, half:]]}


def _coefficients(sw, freqs):
    """k0, the Robin coefficients gamma_p(k) and the ports' beta_p(k)."""
    k0 = 2 * np.pi * np.asarray(freqs) / C0
    gam = np.array([[complex(u.bc.get_gamma(k)) for k in k0] for u in sw.robin])
    beta = np.array([[complex(bc.get_beta(k)) for k in k0] for bc in sw.ports])
    return k0, gam, beta


def _rhs(sw, beta):
    """b_p(k) = -2j beta_p(k) u_p, column f * ports + p."""
    scale = torch.as_tensor((-2j * beta.T).reshape(-1), device="cuda")
    return (sw.u_r.repeat(1, beta.shape[1]) * scale).contiguous()


def _restricted_entries(sw):
    """(row, column, position in the full pattern) of the entries between kept unknowns."""
    ip, ix = sw.plan.indptr, sw.plan.indices[: sw.plan.nnz].long()
    rows = torch.repeat_interleave(torch.arange(len(ip) - 1, device="cuda"), ip[1:] - ip[:-1])
    to = torch.full((len(ip) - 1,), -1, dtype=torch.int64, device="cuda")
    ids = torch.as_tensor(sw.solve_ids, device="cuda")
    to[ids] = torch.arange(len(ids), device="cuda")
    at = torch.nonzero((to[rows] >= 0) & (to[ix] >= 0))[:, 0]
    return to[rows[at]], to[ix[at]], at


def _restricted_dofs(field, ids):
    """(20, tets) restricted unknowns of each tet, -1 where removed."""
    to = np.full(field.n_field, -1, dtype=np.int64)
    to[ids] = np.arange(len(ids))
    return to[field.tet_to_field]


def _levels(field, dofs, n):
    """Breadth-first level of every unknown from the tets at the low end of the longest side."""
    m = field.mesh
    axis = int(np.argmax(np.ptp(m.nodes, axis=1)))
    low = np.isclose(m.nodes[axis], m.nodes[axis].min())
    lev = np.full(n + 1, -1, dtype=np.int64)          # the last entry stands for removed unknowns
    front = np.any(low[m.tets], axis=0)
    done = np.zeros(m.n_tets, dtype=bool)
    k = 0
    while front.any():
        new = np.unique(dofs[:, front])
        new = new[(new >= 0)]
        new = new[lev[new] < 0]
        lev[new] = k
        done |= front
        hit = np.zeros(n + 1, dtype=bool)
        hit[new] = True
        front = np.any(hit[dofs], axis=0) & ~done
        k += 1
    return lev[:n]


def _block_solve(row, col, val, lev, b):
    """A x = b in complex128 by block elimination over the levels (LU with partial pivoting)."""
    dev = b.device
    m = int(lev.max()) + 1
    lv = torch.as_tensor(lev, device=dev)
    order = torch.argsort(lv, stable=True)
    size = torch.bincount(lv, minlength=m)
    off = torch.cumsum(size, 0) - size
    pos = torch.empty_like(order)
    pos[order] = torch.arange(len(order), device=dev)
    local = pos - off[lv]
    sizes = size.tolist()
    by = torch.argsort(lv[row], stable=True)
    row, col, val = row[by], col[by], val[by]
    cut = torch.searchsorted(lv[row].contiguous(), torch.arange(m + 1, device=dev)).tolist()

    def block(i, j):
        s = slice(cut[i], cut[i + 1])
        keep = lv[col[s]] == j
        out = torch.zeros((sizes[i], sizes[j]), dtype=torch.complex128, device=dev)
        out.index_put_((local[row[s][keep]], local[col[s][keep]]), val[s][keep])
        return out

    ids = [order[int(o):int(o) + n] for o, n in zip(off.tolist(), sizes)]
    T, y = [], []
    for i in range(m):
        D, rhs = block(i, i), b[ids[i]]
        if i:
            C = block(i, i - 1)
            D = D - C @ T[-1]
            rhs = rhs - C @ y[-1]
        U = block(i, i + 1) if i + 1 < m else torch.zeros((sizes[i], 0), dtype=torch.complex128, device=dev)
        s = torch.linalg.solve(D, torch.cat([U, rhs], dim=1))
        T.append(s[:, :U.shape[1]].contiguous())
        y.append(s[:, U.shape[1]:].contiguous())
    x = torch.empty_like(b)
    for i in reversed(range(m)):
        v = y[i] if i + 1 == m else y[i] - T[i] @ x[ids[i + 1]]
        x[ids[i]] = v
    return x


def _exact_modes(st):
    """Lowest modes by subspace iteration on the dense shifted matrix, LU with partial pivoting."""
    ce, sigma, k = st["cavity"], st["sigma"], st["modes"]
    ip, ix = ce.sys.pattern()
    n = ce.sys.n
    row = torch.as_tensor(np.repeat(np.arange(n), np.diff(ip)), device="cuda")
    col = torch.as_tensor(ix.astype(np.int64), device="cuda")
    dense = lambda v: torch.zeros((n, n), dtype=torch.complex128, device="cuda").index_put_((row, col), v)  # noqa: E731
    E, B = dense(ce.Er[:, 0]), dense(ce.Br[:, 0])
    lu = torch.linalg.lu_factor(E - sigma * B)
    gen = torch.Generator(device="cuda").manual_seed(1)
    V = torch.randn((n, 6 * k + 10), generator=gen, device="cuda", dtype=torch.float64).to(torch.complex128)
    for it in range(60):
        V = torch.linalg.qr(torch.linalg.lu_solve(*lu, B @ V))[0]
        if it % 3 == 2:      # damp the null space (theta = -1/sigma): a shifted power step
            V = torch.linalg.qr(torch.linalg.lu_solve(*lu, B @ V) + V / sigma)[0]
    W = torch.linalg.lu_solve(*lu, B @ V)
    th = torch.linalg.eigvals(V.conj().T @ W).cpu().numpy()
    lam = sigma + 1.0 / th[np.argsort(-th.real)][:k]
    return {"k0_squared": lam[np.argsort(lam.real)]}


def _exact_assembly(st):
    """E and B from the closed-form element matrices, tets relabelled so that every edge and
    face lists its vertices in ascending order; the face-face mass block keeps the operator's
    own choice of coefficient (it is not symmetric)."""
    m, dev = st["field"].mesh, "cuda"
    put = lambda v: torch.as_tensor(np.asarray(v), device=dev)  # noqa: E731
    T = torch.sort(put(m.tets), dim=0).values
    nT, nN, nE, nF = T.shape[1], m.n_nodes, m.n_edges, m.n_tris
    P = put(m.nodes)[:, T]                                            # (3, 4, nT)
    edges = list(itertools.combinations(range(4), 2))
    faces = list(itertools.combinations(range(4), 3))
    ekey, fkey = put(m.edges[0] * nN + m.edges[1]), put((m.tris[0] * nN + m.tris[1]) * nN + m.tris[2])
    eid = torch.stack([torch.searchsorted(ekey, T[i] * nN + T[j]) for i, j in edges])
    fid = torch.stack([torch.searchsorted(fkey, (T[i] * nN + T[j]) * nN + T[k]) for i, j, k in faces])
    dof = torch.cat([eid, fid + nE, eid + nE + nF, fid + 2 * nE + nF])          # (20, nT)
    e = [P[:, k] - P[:, 0] for k in (1, 2, 3)]
    cr = lambda a, b: torch.linalg.cross(a, b, dim=0)  # noqa: E731
    det = (e[0] * cr(e[1], e[2])).sum(0)
    # 6V grad(lambda_i) up to a common sign; V6 = |det|
    g = [cr(e[1], e[2]), cr(e[2], e[0]), cr(e[0], e[1])]
    G = [-(g[0] + g[1] + g[2])] + g
    V6 = det.abs()
    length = lambda i, j: torch.linalg.norm(P[:, i] - P[:, j], dim=0)  # noqa: E731
    full = st["mat"] == "tensor"
    mul = (lambda M, a: torch.einsum("ijt,jt->it", M.reshape(3, 3, -1), a.to(torch.complex128))) if full else \
        (lambda M, a: M[None] * a)
    X = {(i, j): cr(G[i], G[j]) for i in range(4) for j in range(4) if i != j}
    MG = [mul(st["eps"], v) for v in G]
    MX = {k: mul(st["nu"], v) for k, v in X.items()}
    gg = functools.lru_cache(None)(lambda p, q: (G[p] * MG[q]).sum(0))
    cc = functools.lru_cache(None)(lambda p, q, r, s: (X[p, q] * MX[r, s]).sum(0))

    def v(*idx):
        num = math.prod(math.factorial(idx.count(i)) for i in set(idx))
        return V6 * (num / math.factorial(len(idx) + 3))

    D = torch.zeros((20, 20, nT), dtype=torch.complex128, device=dev)
    F = torch.zeros_like(D)
    # curl-conforming functions: edges L (lam_a grad lam_b - lam_b grad lam_a) lam_{a,b}
    for (i, (A, Bq)), (j, (C, Dq)) in itertools.product(enumerate(edges), repeat=2):
        q = length(A, Bq) * length(C, Dq)
        for r, R in ((0, A), (10, Bq)):
            for s, Sx in ((0, C), (10, Dq)):
                D[i + r, j + s] = 9 * q * cc(A, Bq, C, Dq) * v(R, Sx)
                F[i + r, j + s] = q * (v(Bq, R, Dq, Sx) * gg(A, C) - v(Bq, R, C, Sx) * gg(A, Dq)
                                       - v(A, R, Dq, Sx) * gg(Bq, C) + v(A, R, C, Sx) * gg(Bq, Dq))
    for (i, (A, Bq)), (j, (C, Dq, Fq)) in itertools.product(enumerate(edges), enumerate(faces)):
        ac, ab = length(A, Bq) * length(C, Fq), length(A, Bq) * length(C, Dq)
        I, J, K = cc(A, Bq, C, Fq), cc(A, Bq, Dq, Fq), cc(A, Bq, C, Dq)
        for r, R in ((0, A), (10, Bq)):
            d1 = ac * (-6 * v(R, Dq) * I - 3 * v(R, C) * J - 3 * v(R, Fq) * K)
            d2 = ab * (6 * v(R, Fq) * K + 3 * v(R, Dq) * I - 3 * v(R, C) * J)
            f1 = ac * (v(Bq, R, C, Dq) * gg(A, Fq) - v(Bq, R, Dq, Fq) * gg(A, C)
                       - v(A, R, C, Dq) * gg(Bq, Fq) + v(A, R, Dq, Fq) * gg(Bq, C))
            f2 = ab * (v(Bq, R, Dq, Fq) * gg(A, C) - v(Bq, R, Fq, C) * gg(A, Dq)
                       - v(A, R, Dq, Fq) * gg(Bq, C) + v(A, R, Fq, C) * gg(Bq, Dq))
            for s, dv, fv in ((6, d1, f1), (16, d2, f2)):
                D[i + r, j + s], F[i + r, j + s] = dv, fv
                D[j + s, i + r], F[j + s, i + r] = dv, fv
    for (i, (A, Bq, Eq)), (j, (C, Dq, Fq)) in itertools.product(enumerate(faces), repeat=2):
        l1, l2 = (length(A, Eq), length(A, Bq)), (length(C, Fq), length(C, Dq))
        # curls of the two functions of a face as combinations of the cross products
        rows = ([(2, Bq, (A, Eq)), (1, A, (Bq, Eq)), (1, Eq, (A, Bq))],
                [(-2, Eq, (A, Bq)), (-1, Bq, (A, Eq)), (1, A, (Bq, Eq))])
        cols = ([(2, Dq, (C, Fq)), (1, C, (Dq, Fq)), (1, Fq, (C, Dq))],
                [(-2, Fq, (C, Dq)), (-1, Dq, (C, Fq)), (1, C, (Dq, Fq))])
        for r, s in itertools.product(range(2), repeat=2):
            D[6 + 10 * r + i, 6 + 10 * s + j] = l1[r] * l2[s] * sum(
                p * q * v(x, y) * cc(*ra, *ca) for p, x, ra in rows[r] for q, y, ca in cols[s])
        odd = v(Bq, C, Dq, Fq)
        F[6 + i, 6 + j] = l1[0] * l2[0] * (v(A, Bq, C, Dq) * gg(Eq, Fq) - v(A, Bq, Dq, Fq) * gg(Eq, C)
                                           - odd * gg(A, Fq) + v(Bq, Eq, Dq, Fq) * gg(A, C))
        F[6 + i, 16 + j] = l1[0] * l2[1] * (v(A, Bq, Dq, Fq) * gg(Eq, C) - v(A, Bq, Fq, C) * gg(Eq, Dq)
                                            - v(Bq, Eq, Dq, Fq) * gg(A, C) + v(Bq, Eq, Fq, C) * gg(A, Dq))
        F[16 + i, 6 + j] = l1[1] * l2[0] * (odd * gg(A, Fq) - v(Bq, Eq, Dq, Fq) * gg(A, C)
                                            - v(Eq, A, C, Dq) * gg(Bq, Fq) + v(Eq, A, Dq, Fq) * gg(Bq, C))
        F[16 + i, 16 + j] = l1[1] * l2[1] * (v(Bq, Eq, Dq, Fq) * gg(A, C) - v(Bq, Eq, Fq, C) * gg(A, Dq)
                                             - v(Eq, A, Dq, Fq) * gg(Bq, C) + v(A, C, Eq, Fq) * gg(Bq, Dq))
    D /= V6 ** 4
    F /= V6 ** 2
    N = 2 * nE + 2 * nF
    key = (dof[:, None, :] * N + dof[None, :, :]).reshape(-1)
    uniq, where = torch.unique(key, return_inverse=True)
    out = []
    for M in (D, F):
        s = torch.zeros(len(uniq), dtype=torch.complex128, device=dev)
        out.append(s.index_add_(0, where, M.reshape(-1)))
    return {"E": out[0], "B": out[1]}
