"""A few functionals of every solution column (G = U^T X), at the edges of the kernel's tiles of four
functionals and 128 columns and of its row blocks, against NumPy in extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 65, 20011])
@pytest.mark.parametrize("npo,cols", [(1, 1), (2, 2), (3, 5), (4, 127), (5, 129), (9, 300)])
def test_functionals(n, npo, cols):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from emerge_gb300 import _build
    _build.build()
    from emerge_gb300.solver import functionals
    rng = np.random.default_rng(n + cols)
    U = rng.standard_normal((n, npo)) + 1j * rng.standard_normal((n, npo))
    X = rng.standard_normal((n, cols)) + 1j * rng.standard_normal((n, cols))
    got = functionals(torch.as_tensor(U, device="cuda"), torch.as_tensor(X, device="cuda").T.contiguous().T)
    ref = (U.astype(np.clongdouble).T @ X.astype(np.clongdouble)).astype(complex)
    # n products of a few roundings each, summed in any order
    bound = (n + 8) * 2.0 ** -52 * (np.abs(U).T @ np.abs(X))
    assert np.all(np.abs(got.cpu().numpy() - ref) <= bound)


@pytest.mark.parametrize("n", [1, 65, 20011])
@pytest.mark.parametrize("m,cols", [(1, 1), (3, 4), (44, 4), (300, 10), (5, 2048)])
def test_projection_pieces(n, m, cols):
    """Conjugated functionals on a strided basis, W - V C (more vectors than a round of shared
    memory takes), and column dots."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if n * cols > 1e6:
        n = 65
    from emerge_gb300 import _build
    _build.build()
    from emerge_gb300.solver import column_dots, functionals, sub_product
    rng = np.random.default_rng(n + m)
    rnd = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    V, W, C = rnd(n, m + 3), rnd(n, cols), rnd(m, cols)
    Vd, Wd, Cd = (torch.as_tensor(a, device="cuda") for a in (V, W, C))
    V = V[:, 2:2 + m]
    wide = lambda a: a.astype(np.clongdouble)  # noqa: E731
    got = functionals(Vd[:, 2:2 + m], Wd, conj=True).cpu().numpy()
    assert np.all(np.abs(got - wide(V).conj().T @ wide(W)) <= (n + 8) * 2.0 ** -52 * (np.abs(V).T @ np.abs(W)))
    got = sub_product(Wd, Vd[:, 2:2 + m], Cd).cpu().numpy()
    assert np.all(np.abs(got - (wide(W) - wide(V) @ wide(C))) <= (m + 8) * 2.0 ** -52 * (np.abs(W) + np.abs(V) @ np.abs(C)))
    got = column_dots(Wd, Wd).cpu().numpy()
    assert np.all(np.abs(got - (wide(W).conj() * wide(W)).sum(axis=0)) <= (n + 8) * 2.0 ** -52 * (np.abs(W) ** 2).sum(axis=0))
