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


def _chain(S, x, parts):
    """S x by chains of FP32 products and sums over K in ``parts`` consecutive parts, the parts added in order."""
    import torch
    n, K, c = S.shape[0], S.shape[1], x.shape[1]
    step = -(-K // parts)
    Sp = torch.zeros((n, parts * step), dtype=torch.complex64, device=S.device)
    xp = torch.zeros((parts * step, c), dtype=torch.complex64, device=S.device)
    Sp[:, :K], xp[:K] = S, x
    cols = [a.contiguous() for a in (Sp.real.reshape(n, parts, step).permute(2, 1, 0)[..., None],
                                     Sp.imag.reshape(n, parts, step).permute(2, 1, 0)[..., None])]
    rows = [a.reshape(parts, step, 1, c).transpose(0, 1).contiguous() for a in (xp.real, xp.imag)]
    re, im = (torch.zeros((parts, n, c), dtype=torch.float32, device=S.device) for _ in range(2))
    for sr, si, xr, xi in zip(cols[0], cols[1], rows[0], rows[1]):
        re.addcmul_(sr, xr).addcmul_(si, xi, value=-1.0)
        im.addcmul_(sr, xi).addcmul_(si, xr)
    out = torch.complex(re[0], im[0])
    for p in range(1, parts):
        out = out + torch.complex(re[p], im[p])
    return out.to(torch.complex128)


@pytest.mark.parametrize("n,cols", [(300, 16), (300, 70), (941, 130), (1380, 65), (2000, 16), (2000, 48)])
def test_products_are_as_accurate_as_fp32_chains(torch_cuda, n, cols):
    """A solve's product of the stored FP32 inverse is no further from 64 bits than chains of FP32 FMAs over
    K / parts, with parts for two tiles a multiprocessor and 256 of K or more each."""
    torch = torch_cuda
    from emerge_gb300.solver import RestrictedSystem, SlabFactor
    ip = torch.arange(0, n * n + 1, n, dtype=torch.int64, device="cuda")
    ix = torch.arange(n, dtype=torch.int32, device="cuda").repeat(n)
    slab = SlabFactor(RestrictedSystem(ip, ix, n * n, np.arange(n)), np.arange(n))
    gen = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.view_as_complex(torch.randn((*s, 2), generator=gen, device="cuda", dtype=torch.float64))  # noqa: E731
    A = rnd(n, n) / (2 * n) ** 0.5 + 1.2 * torch.eye(n, device="cuda")
    slab.factor(A.reshape(-1, 1).contiguous(), [0], "fp32")
    eye = torch.eye(n, dtype=torch.complex128, device="cuda")
    S = torch.cat([slab.apply(eye[:, c:c + 1].contiguous(), [0]) for c in range(n)], dim=1)   # one column: exact
    x = rnd(n, cols).to(torch.complex64).to(torch.complex128)
    for v in (x, torch.complex(x.real.abs(), x.imag.abs())):
        ref = S @ v
        tiles = -(-n // 128) if cols <= 16 else -(-n // 64) * -(-cols // 64)
        parts = max(1, min(-(-304 // tiles), n // 256, 8))
        err = torch.linalg.norm(slab.apply(v, [0] * cols) - ref)
        assert float(err) <= float(torch.linalg.norm(_chain(S, v, parts) - ref))
