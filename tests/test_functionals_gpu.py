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
