"""FP64 slab factors from FP16 digits on the tensor cores: one dense block at the tile edges, rows
and columns scaled over many orders of magnitude, and non-finite entries.

The inverse of a well-conditioned n x n block (condition below 100 after scaling) has a relative
error of a few n eps; scaling rows and columns by powers of two changes no digit of it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from emerge_gb300 import _build
    _build.build()
    return torch


def _dense_system(torch, n):
    from emerge_gb300.solver import RestrictedSystem, SlabFactor
    ip = torch.arange(0, n * n + 1, n, dtype=torch.int64, device="cuda")
    ix = torch.arange(n, dtype=torch.int32, device="cuda").repeat(n)
    sysr = RestrictedSystem(ip, ix, n * n, np.arange(n))
    slab = SlabFactor(sysr, np.arange(n))          # all unknowns are seeds: one slab
    assert slab.info()["slabs"] == 1
    return sysr, slab


def _matrix(torch, n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.view_as_complex(torch.randn((n, n, 2), generator=gen, device="cuda", dtype=torch.float64)) / (2 * n) ** 0.5
    return A + 3.0 * torch.eye(n, device="cuda")


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 96, 127, 128, 129, 191, 193, 320])
@pytest.mark.parametrize("tensor_cores", [True, False])
def test_dense_inverse(torch_cuda, n, tensor_cores):
    torch = torch_cuda
    sysr, slab = _dense_system(torch, n)
    A = _matrix(torch, n, n)
    slab.set_factor_tensor_cores(tensor_cores)
    slab.factor(A.reshape(-1, 1).contiguous(), [0], "fp64")
    X = slab.apply(torch.eye(n, dtype=torch.complex128, device="cuda"), [0] * n)
    R = A @ X - torch.eye(n, device="cuda")
    assert float(torch.linalg.norm(R, ord=2)) <= 100 * n * EPS
    assert slab.info()["perturbed_pivots"] == 0


def test_scaled_rows_and_columns(torch_cuda):
    torch = torch_cuda
    n = 200
    sysr, slab = _dense_system(torch, n)
    A = _matrix(torch, n, 5)
    rng = np.random.default_rng(2)
    # the largest spread that keeps every pivot above the 1e-13 of the tile maximum where it is replaced
    dr = torch.as_tensor(2.0 ** rng.integers(-8, 9, n), device="cuda")
    dc = torch.as_tensor(2.0 ** rng.integers(-8, 9, n), device="cuda")
    S = dr[:, None] * A * dc[None, :]
    slab.factor(S.reshape(-1, 1).contiguous(), [0], "fp64")
    X = slab.apply(torch.eye(n, dtype=torch.complex128, device="cuda"), [0] * n)
    assert slab.info()["perturbed_pivots"] == 0
    R = A @ (dc[:, None] * X * dr[None, :]) - torch.eye(n, device="cuda")
    assert float(torch.linalg.norm(R, ord=2)) <= 1e5 * n * EPS    # row scaling changes the pivots of a tile


def test_two_factors_of_one_launch(torch_cuda):
    torch = torch_cuda
    n = 130
    sysr, slab = _dense_system(torch, n)
    A, B = _matrix(torch, n, 8), _matrix(torch, n, 9)
    slab.factor(torch.stack([A.reshape(-1), B.reshape(-1)], dim=1).contiguous(), [1, 0], "fp64")
    eye = torch.eye(n, dtype=torch.complex128, device="cuda")
    for f, M in ((0, B), (1, A)):
        assert float(torch.linalg.norm(M @ slab.apply(eye, [f] * n) - eye, ord=2)) <= 100 * n * EPS


def test_non_finite_entries_stay_visible(torch_cuda):
    """A non-finite entry outside the first pivot tile gives non-finite results, not finite wrong ones."""
    torch = torch_cuda
    n = 150
    sysr, slab = _dense_system(torch, n)
    A = _matrix(torch, n, 11)
    A[100, 20] = complex(float("inf"), 0.0)
    slab.factor(A.reshape(-1, 1).contiguous(), [0], "fp64")
    X = slab.apply(torch.ones((n, 1), dtype=torch.complex128, device="cuda"), [0])
    assert not bool(torch.isfinite(torch.view_as_real(X)).all())


@pytest.mark.parametrize("n", [40, 64, 130])
@pytest.mark.parametrize("cond", [1e2, 1e4, 1e7, 1e11])
def test_ill_conditioned_tiles(torch_cuda, n, cond):
    """Tiles that the Newton steps from an FP32 inverse take, and those left to the exchange steps."""
    torch = torch_cuda
    sysr, slab = _dense_system(torch, n)
    U, V = (torch.linalg.qr(_matrix(torch, n, s) - 3.0 * torch.eye(n, device="cuda"))[0] for s in (21, 22))
    d = torch.logspace(0, -np.log10(cond), n, dtype=torch.float64, device="cuda")
    A = (U * d) @ V
    slab.factor(A.reshape(-1, 1).contiguous(), [0], "fp64")
    X = slab.apply(torch.eye(n, dtype=torch.complex128, device="cuda"), [0] * n)
    R = A @ X - torch.eye(n, device="cuda")
    # pivots of a tile may be smaller than those of the whole matrix: a factor of its growth
    assert float(torch.linalg.norm(R, ord=2)) <= 1000 * n * cond * EPS
    assert slab.info()["perturbed_pivots"] == 0


@pytest.mark.parametrize("n", [10, 64, 100])
def test_zero_pivot_is_replaced(torch_cuda, n):
    torch = torch_cuda
    sysr, slab = _dense_system(torch, n)
    d = torch.full((n,), 3.0 + 1.0j, dtype=torch.complex128, device="cuda")
    d[5] = 0.0
    slab.factor(torch.diag(d).reshape(-1, 1).contiguous(), [0], "fp64")
    X = slab.apply(torch.eye(n, dtype=torch.complex128, device="cuda"), [0] * n)
    assert slab.info()["perturbed_pivots"] == 1
    keep = [i for i in range(n) if i != 5]
    assert torch.allclose(torch.diag(X)[keep], 1.0 / d[keep], rtol=1e-14, atol=0.0)
    assert bool(torch.isfinite(torch.view_as_real(X)).all())


def _product_of(torch, B, C, tensor_cores):
    """B C by a factorization: the inverse of [[1, B, 0], [0, 1, C], [0, 0, 1]] holds it."""
    n = 192
    M = torch.eye(n, dtype=torch.complex128)
    M[:64, 64:128], M[64:128, 128:] = torch.as_tensor(B), torch.as_tensor(C)
    _, slab = _dense_system(torch, n)
    slab.set_factor_tensor_cores(tensor_cores)
    slab.factor(M.cuda().reshape(-1, 1).contiguous(), [0], "fp64")
    return slab.apply(torch.eye(n, dtype=torch.complex128, device="cuda"), [0] * n).cpu().numpy()[:64, 128:]


@pytest.mark.parametrize("tensor_cores", [True, False])
@pytest.mark.parametrize("spread", [0.0, 2.0 ** -40, 2.0 ** -30, 2.0 ** -21, 2.0 ** -12])
def test_repeated_values(torch_cuda, tensor_cores, spread):
    """Products of rows and columns of one value each, or of values that differ in their low digits
    only: no digit sum may leave the integers that an accumulator holds."""
    torch = torch_cuda
    rng = np.random.default_rng(3)
    c = np.r_[0.92371687, 1.0 - 2.0 ** -30, rng.uniform(0.5, 1.0, 62)]
    vary = lambda: 1.0 + spread * rng.uniform(-1.0, 1.0, (64, 64))  # noqa: E731
    B = c[:, None] * vary() + 1j * c[:, None] * vary()
    C = c[None, :] * vary() + 1j * c[None, :] * vary()
    X = _product_of(torch, B, C, tensor_cores)
    wide = lambda a: a.astype(np.clongdouble)  # noqa: E731
    # a chain of 64 complex products of four roundings: at most 130 of half an eps each (and one for the result)
    assert np.all(np.abs(X - wide(B) @ wide(C)) <= 131 * EPS / 2 * (np.abs(B) @ np.abs(C)))


@pytest.mark.parametrize("scale", [9e-155, 1.0, 1.2e154])
def test_pivots_at_the_ends_of_the_range(torch_cuda, scale):
    """Tiles for the exchange steps (one zero pivot, one pair that is singular in FP32) whose squared
    pivots are subnormal or have a subnormal reciprocal."""
    torch = torch_cuda
    n = 40
    sysr, slab = _dense_system(torch, n)
    A = np.eye(n) + 0.01 * np.random.default_rng(4).uniform(-1, 1, (n, n))
    A[5], A[:, 5] = 0.0, 0.0
    keep = np.delete(np.arange(n), 5)
    if scale >= 1.0:
        A[[7, 8]], A[:, [7, 8]] = 0.0, 0.0
        A[7:9, 7:9] = [[1.0, 1.0], [1.0, 1.0 + 2.0 ** -24]]
    slab.factor(torch.as_tensor(scale * A + 0j, device="cuda").reshape(-1, 1).contiguous(), [0], "fp64")
    X = slab.apply(torch.eye(n, dtype=torch.complex128, device="cuda"), [0] * n).cpu().numpy()
    assert slab.info()["perturbed_pivots"] == 1
    K = A[np.ix_(keep, keep)]
    Y, apart = scale * X[np.ix_(keep, keep)], np.isin(keep, (7, 8)) & (scale >= 1.0)
    ref = np.linalg.inv(K)
    # without the pair, whose rows and columns are apart: condition below 3, a subnormal |pivot|^2 has 50 bits
    assert np.all(np.abs(Y - ref)[~apart] <= 64 * n * EPS * np.max(np.abs(ref), axis=1)[~apart, None])
    # the pair, condition 2^26: the residual of each entry against the magnitudes of its products
    assert np.all(np.abs(K @ Y - np.eye(n - 1)) <= 64 * n * EPS * (np.abs(K) @ np.abs(Y)) + 64 * n * EPS)


@pytest.mark.parametrize("n", [1, 17, 40, 64])
@pytest.mark.parametrize("cond", [1e1, 1e2, 1e3, 1e4])
def test_tile_inverse_is_near_its_rounding(torch_cuda, n, cond):
    """One pivot tile from its FP32 inverse: the residual is formed nearly exactly, so the error is the
    rounding of the result, not that times the condition."""
    torch = torch_cuda
    sysr, slab = _dense_system(torch, n)
    U, V = (torch.linalg.qr(_matrix(torch, n, s) - 3.0 * torch.eye(n, device="cuda"))[0] for s in (31, 32))
    A = (U * torch.logspace(0, -np.log10(cond), n, dtype=torch.float64, device="cuda")) @ V
    slab.factor(A.reshape(-1, 1).contiguous(), [0], "fp64")
    X = slab.apply(torch.eye(n, dtype=torch.complex128, device="cuda"), [0] * n).cpu().numpy()
    T = A.cpu().numpy().astype(np.clongdouble)
    ref = np.linalg.inv(A.cpu().numpy()).astype(np.clongdouble)
    for _ in range(3):
        ref = ref + ref @ (np.eye(n) - T @ ref)
    # three or four sums of half an eps of the largest entry and products with a residual below 0.1
    assert np.max(np.abs(X - ref)) <= 8 * EPS * np.max(np.abs(ref))
