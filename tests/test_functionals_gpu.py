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


def _block(torch, *shape, seed=0, device="cuda"):
    gen = torch.Generator(device="cpu").manual_seed(seed)
    return torch.view_as_complex(torch.randn((*shape, 2), generator=gen, dtype=torch.float64)).to(device)


def test_lazily_conjugated_blocks():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from emerge_gb300.solver import column_dots, functionals, sub_product
    V, W, C = _block(torch, 65, 3), _block(torch, 65, 4, seed=1), _block(torch, 3, 4, seed=2)
    near = lambda a, b: bool(((a - b).abs() <= 80 * 2.0 ** -52 * 100).all())  # noqa: E731
    for view in (torch.conj, torch._neg_view, lambda t: torch._neg_view(t.conj())):
        v, w, c = view(V), view(W), view(C)
        vr, wr, cr = (t.resolve_conj().resolve_neg().clone() for t in (v, w, c))
        assert near(functionals(v, W), vr.T @ W) and near(functionals(V, w), V.T @ wr)
        assert near(functionals(v, w, conj=True), vr.conj().T @ wr)
        assert near(column_dots(w, W), (wr.conj() * W).sum(dim=0)) and near(column_dots(W, w), (W.conj() * wr).sum(dim=0))
        assert near(sub_product(w, v, c), wr - vr @ cr)


def test_more_columns_than_the_kernel_takes():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from emerge_gb300.solver import sub_product
    V, W, C = _block(torch, 17, 3), _block(torch, 17, 2049, seed=1), _block(torch, 3, 2049, seed=2)
    assert torch.allclose(sub_product(W, V, C), W - V @ C, rtol=0.0, atol=1e-13)


def test_what_torch_refuses_stays_refused():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from emerge_gb300.solver import column_dots, functionals, sub_product
    V, W, C = _block(torch, 65, 3), _block(torch, 65, 4, seed=1), _block(torch, 3, 4, seed=2)
    for call in (lambda: functionals(V, W[:60]), lambda: functionals(V[:60], W), lambda: functionals(V, W.to(torch.complex64)),
                 lambda: functionals(V.cpu(), W), lambda: column_dots(W, W[:60]), lambda: column_dots(W, W.cpu()),
                 lambda: sub_product(W, V, C[:2]), lambda: sub_product(W, V, C[:, :3]), lambda: sub_product(W[:60], V, C),
                 lambda: sub_product(W, V.to(torch.complex64), C), lambda: sub_product(W, V, C.cpu())):
        with pytest.raises(RuntimeError):
            call()
    # and what it computes is computed
    V4, W4, C4 = (t.to(torch.complex64) for t in (V, W, C))
    assert torch.allclose(functionals(V4, W4), V4.T @ W4) and torch.allclose(sub_product(W4, V4, C4), W4 - V4 @ C4)
    assert torch.allclose(column_dots(W4, W), (W4.conj() * W).sum(dim=0))
    assert torch.allclose(column_dots(W, W[:1]), (W.conj() * W[:1]).sum(dim=0))
    assert torch.allclose(functionals(V.real, W.real), V.real.T @ W.real)
    g = W.clone().requires_grad_()
    column_dots(g, g).real.sum().backward()
    assert torch.allclose(g.grad, 2 * W)
