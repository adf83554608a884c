"""Kernels of the restricted solves at the sizes where their dispatch changes: forming A(k) with
and without port matrices, products with few and many columns, and the Gram-Schmidt dots of a
solve, against plain FP64 torch.

Tolerance of a sum of m products: each result is within (m + 2) eps of the sum of magnitudes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.fixture(scope="module")
def system():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from emerge_gb300 import _build
    _build.build()
    from emerge_gb300.solver import RestrictedSystem
    import scipy.sparse as sp
    rng = np.random.default_rng(7)
    n = 331
    M = (sp.random(n, n, 0.05, random_state=3, format="csr") + sp.eye(n)).tocsr()
    M.sort_indices()
    ids = np.sort(rng.choice(n, 301, replace=False))
    put = lambda v: torch.as_tensor(v, device="cuda")  # noqa: E731
    sysr = RestrictedSystem(put(M.indptr.astype(np.int64)), put(M.indices.astype(np.int32)), M.nnz, ids)
    keep = np.full(n, -1)
    keep[ids] = np.arange(len(ids))
    row = np.repeat(np.arange(n), np.diff(M.indptr))
    at = np.flatnonzero((keep[row] >= 0) & (keep[M.indices] >= 0))
    return sysr, put(at), put(keep[row[at]]), put(keep[M.indices[at]])


def _complex(gen, *shape):
    import torch
    return torch.view_as_complex(torch.randn((*shape, 2), generator=gen, device="cuda", dtype=torch.float64))


@pytest.mark.parametrize("ports", [0, 1, 4, 6])
@pytest.mark.parametrize("Bm", [1, 3, 64, 300])
def test_form(system, ports, Bm):
    import torch
    sysr, at, _, _ = system
    gen = torch.Generator(device="cuda").manual_seed(Bm + ports)
    E, B = _complex(gen, sysr.nnz_full), _complex(gen, sysr.nnz_full)
    k2 = np.random.default_rng(1).uniform(0, 5, Bm)
    P = gam = None
    if ports:
        P = _complex(gen, ports, sysr.nnz_full) * (torch.arange(sysr.nnz_full, device="cuda") % 7 == 0)
        gam = _complex(gen, ports, Bm).cpu().numpy()
    A = sysr.form(E, B, k2, P, gam)
    q = torch.as_tensor(k2, device="cuda")
    ref = E[at][:, None] - q * B[at][:, None]
    mag = E[at].abs()[:, None] + q * B[at].abs()[:, None]
    if ports:
        g = torch.as_tensor(gam, device="cuda")
        ref = ref + P[:, at].T @ g
        mag = mag + P[:, at].T.abs().to(torch.float64) @ g.abs()
    assert bool(((A - ref).abs() <= (2 * ports + 4) * EPS * mag).all())


def test_form_with_a_non_finite_gamma(system):
    """0 * inf stays NaN: entries off the port keep what a full product gives."""
    import torch
    sysr, _, _, _ = system
    E = torch.ones(sysr.nnz_full, dtype=torch.complex128, device="cuda")
    P = torch.zeros((1, sysr.nnz_full), dtype=torch.complex128, device="cuda")
    A = sysr.form(E, E, [1.0, 2.0], P, np.array([[1.0, np.inf]], dtype=complex))
    assert bool(torch.isfinite(A[:, 0].abs()).all()) and bool(torch.isnan(A[:, 1].abs()).all())


@pytest.mark.parametrize("Bc", [1, 2, 3, 4, 5, 8, 9, 129])
@pytest.mark.parametrize("residual", [False, True])
def test_spmv(system, Bc, residual):
    import torch
    sysr, _, row, col = system
    gen = torch.Generator(device="cuda").manual_seed(Bc)
    A, X = _complex(gen, sysr.nnz, 3), _complex(gen, sysr.n, Bc)
    b = _complex(gen, sysr.n, Bc) if residual else None
    cmat = (torch.arange(Bc, device="cuda") % 3).to(torch.int32)
    Y = sysr.spmv(A, X, cmat, b)
    prod = A[:, cmat.long()] * X[col]
    ref = torch.zeros_like(X).index_add_(0, row, prod)
    mag = torch.zeros(X.shape, dtype=torch.float64, device="cuda").index_add_(0, row, prod.abs())
    if residual:
        ref, mag = b - ref, mag + b.abs()
    assert bool(((Y - ref).abs() <= 70 * EPS * mag).all())     # rows hold at most 40 entries


@pytest.mark.parametrize("Bc", [1, 3, 31, 32, 33, 128, 129, 257])
def test_gmres_columns(system, Bc):
    """A diagonally dominant system: every column count takes the same few steps to 1e-12."""
    import torch
    sysr, _, row, col = system
    gen = torch.Generator(device="cuda").manual_seed(Bc)
    A = 0.02 * _complex(gen, sysr.nnz, 1)
    A[row == col] += 1.0
    x = _complex(gen, sysr.n, Bc)
    cmat = torch.zeros(Bc, dtype=torch.int32, device="cuda")
    b = sysr.spmv(A, x, cmat)
    got, its, res = sysr.gmres(A, sysr.ilu0(A), b, cmat, restart=40, max_iter=40, tol=1e-12)
    assert res.max() <= 1e-12 and its.max() <= 20
    # |I - A| < 1/2 row-wise, so the error is at most twice the residual in the 2-norm
    assert float(torch.linalg.norm(got - x) / torch.linalg.norm(b)) <= 4e-12
