"""FP32 slab factors of one dense block at the edges of the row panel's 16-column strips, the 64-wide
pivot tiles and the 128-row update tiles, and the next pivot tile formed by the row panel.

The inverse of a well-conditioned n x n block (condition below 100 after scaling) has a relative
error of a few n eps.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -23


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from emerge_gb300 import _build
    _build.build()
    return torch


@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 79, 80, 81, 127, 128, 129, 145, 193, 321])
@pytest.mark.parametrize("factors", [1, 2])
def test_dense_inverse(torch_cuda, n, factors):
    torch = torch_cuda
    from emerge_gb300.solver import RestrictedSystem, SlabFactor
    ip = torch.arange(0, n * n + 1, n, dtype=torch.int64, device="cuda")
    ix = torch.arange(n, dtype=torch.int32, device="cuda").repeat(n)
    sysr = RestrictedSystem(ip, ix, n * n, np.arange(n))
    slab = SlabFactor(sysr, np.arange(n))          # all unknowns are seeds: one slab
    gen = torch.Generator(device="cuda").manual_seed(n)
    A = torch.view_as_complex(torch.randn((factors, n, n, 2), generator=gen, device="cuda", dtype=torch.float64))
    A = A / (2 * n) ** 0.5 + 3.0 * torch.eye(n, device="cuda")
    slab.factor(A.reshape(factors, -1).T.contiguous(), list(range(factors)), "fp32")
    eye = torch.eye(n, dtype=torch.complex128, device="cuda")
    for f in range(factors):
        R = A[f] @ slab.apply(eye, [f] * n) - eye
        assert float(torch.linalg.norm(R, ord=2)) <= 100 * n * EPS
    assert slab.info()["perturbed_pivots"] == 0
