"""Slab solves of every column count at which the dense product changes (rows of few columns,
tensor-core tiles, column tiles of 64), one and two factors, odd slab widths.

The products work on the same factors, so the error of a solve is the factor's: each column
count must be within twice the error of single columns (FP32), or within 1e-9 (FP64).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from emerge_gb300 import _build
    _build.build()
    from emerge_gb300.freq import Assembler
    from emerge_gb300.geometry import straight_waveguide
    from emerge_gb300.solver import FrequencySweep, RestrictedSystem, SlabFactor, locality_key
    p = straight_waveguide(5e-3)
    sw = FrequencySweep(Assembler(), p.field, p.er, p.ur, p.bcs)
    k0, gam, _ = sw._coeffs([9.1e9, 10.7e9])
    # without every 29th unknown some slabs are odd: their rows are not 16-byte aligned
    ids = np.delete(sw.solve_ids, np.arange(0, len(sw.solve_ids), 29))
    sysr = RestrictedSystem(sw.plan.indptr, sw.plan.indices[: sw.plan.nnz], sw.plan.nnz, ids)
    A = sysr.form(sw.E, sw.B, k0 ** 2, sw.P, gam)
    return torch, sysr, A, SlabFactor(sysr, None, locality_key(p.field, ids))


COLUMNS = [1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 33, 48, 63, 64, 65, 130]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_column_counts(system, precision):
    torch, sysr, A, slab = system
    off, _ = slab.levels()
    assert np.any(np.diff(off) % 2 == 1)
    slab.factor(A, [0, 1], precision)
    gen = torch.Generator(device="cuda").manual_seed(3)
    n = sysr.n
    x = torch.view_as_complex(torch.randn((n, 2 * max(COLUMNS), 2), generator=gen, device="cuda", dtype=torch.float64))
    cm = torch.zeros(x.shape[1], dtype=torch.int32, device="cuda")
    cm[1::2] = 1                                   # column c belongs to matrix c % 2
    b = sysr.spmv(A, x, cm)
    err = lambda y, ref: (torch.linalg.norm(y - ref, dim=0) / torch.linalg.norm(ref, dim=0)).cpu().numpy()  # noqa: E731
    single = max(err(slab.apply(b[:, c:c + 1], [c % 2]), x[:, c:c + 1])[0] for c in range(12))
    limit = 2 * single if precision == "fp32" else 1e-9
    for cols in COLUMNS:
        one = torch.arange(0, 2 * cols, 2, device="cuda")            # one group
        two = torch.cat([one, one + 1])                                # two groups, one per factor
        for pick, fac in ((one, [0] * cols), (two, [0] * cols + [1] * cols)):
            e = err(slab.apply(b[:, pick], fac), x[:, pick])
            assert e.max() <= limit, (cols, len(fac), e.max(), limit)


def test_split_settings_agree(system):
    """The K split changes the order of the sum only."""
    torch, sysr, A, slab = system
    slab.factor(A, [0], "fp32")
    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.view_as_complex(torch.randn((sysr.n, 20, 2), generator=gen, device="cuda", dtype=torch.float64))
    b = sysr.spmv(A, x, torch.zeros(20, dtype=torch.int32, device="cuda"))
    errs = []
    for splits in (1, 2, 4, 8, 16):
        slab.set_max_splits(splits)
        y = slab.apply(b, [0] * 20)
        assert torch.equal(torch.view_as_real(y), torch.view_as_real(slab.apply(b, [0] * 20)))
        errs.append(float(torch.linalg.norm(y - x) / torch.linalg.norm(x)))
    slab.set_max_splits(8)
    assert max(errs) <= 2 * min(errs)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("cols", [2, 24])
def test_replayed_cycles(system, precision, cols):
    """Cycles of one step replay a captured graph of the chained solve launches."""
    torch, sysr, A, slab = system
    slab.factor(A, [0], precision)
    gen = torch.Generator(device="cuda").manual_seed(5)
    b = torch.view_as_complex(torch.randn((sysr.n, cols, 2), generator=gen, device="cuda", dtype=torch.float64))
    cm = torch.ones(cols, dtype=torch.int32, device="cuda")          # the other frequency's matrix: several cycles
    x, its, res = slab.gmres(A, b, cm, [0] * cols, tol=1e-3, restart=1, max_iter=12)
    y, its_y, res_y = slab.gmres(A, b, cm, [0] * cols, tol=1e-3, restart=1, max_iter=12)
    assert its.min() > 1 and np.array_equal(its, its_y)
    assert torch.equal(torch.view_as_real(x), torch.view_as_real(y))
    true = (torch.linalg.norm(b - sysr.spmv(A, x, cm), dim=0) / torch.linalg.norm(b, dim=0)).cpu().numpy()
    assert np.all(np.abs(true - res) <= 1e-9)                        # the reported residual is that of x


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_factor_counts(system, precision):
    """The Schur products take 2, 4 or 8 columns a block with the number of factors, and with a
    hundred the rows in parts; no sum changes its order."""
    torch, sysr, A, slab = system
    gen = torch.Generator(device="cuda").manual_seed(6)
    b = torch.view_as_complex(torch.randn((sysr.n, 2, 2), generator=gen, device="cuda", dtype=torch.float64))
    slab.factor(A, [0, 1], precision)
    ref = torch.view_as_real(slab.apply(b, [0, 1]))
    for F in (3, 6, 12, 30, 100):
        slab.factor(A, [0, 1] + [0] * (F - 3) + [1], precision)
        for fac in ([0, 1], [0, F - 1], [F - 2 if F > 3 else 0, 1]):
            assert torch.equal(torch.view_as_real(slab.apply(b, fac)), ref), F


def test_split_settings_agree_on_tiles(system):
    """The same with more columns than the row blocks take: the tensor-core tiles' K split."""
    torch, sysr, A, slab = system
    slab.factor(A, [0], "fp32")
    gen = torch.Generator(device="cuda").manual_seed(7)
    x = torch.view_as_complex(torch.randn((sysr.n, 70, 2), generator=gen, device="cuda", dtype=torch.float64))
    b = sysr.spmv(A, x, torch.zeros(70, dtype=torch.int32, device="cuda"))
    errs = []
    for splits in (1, 2, 4, 8, 16):
        slab.set_max_splits(splits)
        y = slab.apply(b, [0] * 70)
        assert torch.equal(torch.view_as_real(y), torch.view_as_real(slab.apply(b, [0] * 70)))
        errs.append(float(torch.linalg.norm(y - x) / torch.linalg.norm(x)))
    slab.set_max_splits(8)
    assert max(errs) <= 2 * min(errs)


@pytest.mark.parametrize("n", [1, 3, 7, 8, 9, 63, 129, 515, 1217])
def test_row_blocks(system, n):
    """Row blocks on one slab of a known inverse: widths and column counts around their tiles."""
    torch = system[0]
    from emerge_gb300.solver import RestrictedSystem, SlabFactor
    ip = torch.arange(0, n * n + 1, n, dtype=torch.int64, device="cuda")
    ix = torch.arange(n, dtype=torch.int32, device="cuda").repeat(n)
    slab = SlabFactor(RestrictedSystem(ip, ix, n * n, np.arange(n)), np.arange(n))
    gen = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.view_as_complex(torch.randn((*s, 2), generator=gen, device="cuda", dtype=torch.float64))  # noqa: E731
    A = [rnd(n, n) / (2 * n) ** 0.5 + 3.0 * torch.eye(n, device="cuda") for _ in range(3)]
    slab.factor(torch.stack([a.reshape(-1) for a in A], dim=1).contiguous(), [0, 1, 2], "fp32")
    for cols in (1, 4, 8, 9, 16, 17, 24, 31, 32, 33, 48, 49, 64):
        for G in (1, 2, 3):
            b = rnd(n, cols * G)
            y = slab.apply(b, sum(([g] * cols for g in range(G)), []))
            for g in range(G):
                r = A[g] @ y[:, g * cols:(g + 1) * cols] - b[:, g * cols:(g + 1) * cols]
                # inverse and product: relative errors of a few n eps, condition below 100
                assert float(torch.linalg.norm(r)) <= 200 * n * 2.0 ** -23 * float(torch.linalg.norm(b))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("cols", [2, 24])
def test_solves_in_a_row_on_another_stream(system, precision, cols):
    """Solves with other columns' factors follow each other on a stream without a wait: each works with
    its own column tables."""
    torch, sysr, A, slab = system
    slab.factor(A, [0, 1], precision)
    gen = torch.Generator(device="cuda").manual_seed(8)
    b = torch.view_as_complex(torch.randn((sysr.n, cols, 2), generator=gen, device="cuda", dtype=torch.float64))
    facs = [[0] * cols, [1] * cols, [0] + [1] * (cols - 1), [c % 2 for c in range(cols)]]
    refs = []
    for fac in facs:
        refs.append(torch.view_as_real(slab.apply(b, fac)))
        torch.cuda.synchronize()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = [slab.apply(b, facs[i % 4]) for i in range(12)]
    side.synchronize()
    for i, y in enumerate(got):
        assert torch.equal(torch.view_as_real(y), refs[i % 4]), i


@pytest.mark.parametrize("precision,cols", [("fp32", 1), ("fp32", 20), ("fp64", 20)])
def test_a_solve_does_not_wait_for_the_gpu(system, precision, cols):
    """A product by rows or row blocks has no status to read: the call returns while earlier work runs."""
    torch, sysr, A, slab = system
    slab.factor(A, [0], precision)
    b = torch.ones((sysr.n, cols), dtype=torch.complex128, device="cuda")
    ref = slab.apply(b, [0] * cols)                # work space and kernels are there
    x = torch.ones((8192, 8192), device="cuda")
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    for _ in range(100):                           # over 100 ms of FP32 products
        x = x @ x * 0.0
    done.record()
    y = slab.apply(b, [0] * cols)
    assert not done.query()
    assert torch.equal(torch.view_as_real(y), torch.view_as_real(ref))


@pytest.mark.parametrize("n", [1473, 1505])
def test_narrow_tiles_of_wide_slabs(system, n):
    """Four groups of up to 16 columns on slabs so wide that the 128 x 16 tiles serve them."""
    torch = system[0]
    from emerge_gb300.solver import RestrictedSystem, SlabFactor
    ip = torch.arange(0, n * n + 1, n, dtype=torch.int64, device="cuda")
    ix = torch.arange(n, dtype=torch.int32, device="cuda").repeat(n)
    slab = SlabFactor(RestrictedSystem(ip, ix, n * n, np.arange(n)), np.arange(n))
    gen = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.view_as_complex(torch.randn((*s, 2), generator=gen, device="cuda", dtype=torch.float64))  # noqa: E731
    A = [rnd(n, n) / (2 * n) ** 0.5 + 3.0 * torch.eye(n, device="cuda") for _ in range(4)]
    slab.factor(torch.stack([a.reshape(-1) for a in A], dim=1).contiguous(), [0, 1, 2, 3], "fp32")
    for sizes in ([4] * 4, [8] * 4, [9, 4, 1, 16], [16] * 4):
        b = rnd(n, sum(sizes))
        y = slab.apply(b, sum(([g] * c for g, c in enumerate(sizes)), []))
        assert torch.equal(torch.view_as_real(y), torch.view_as_real(slab.apply(b, sum(([g] * c for g, c in enumerate(sizes)), []))))
        for g, c in enumerate(sizes):
            col = sum(sizes[:g])
            r = A[g] @ y[:, col:col + c] - b[:, col:col + c]
            # inverse and product: relative errors of a few n eps, condition below 100
            assert float(torch.linalg.norm(r)) <= 200 * n * 2.0 ** -23 * float(torch.linalg.norm(b[:, col:col + c]))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_a_solve_cannot_be_captured(system, precision):
    """A captured solve would read the caller's column tables at every replay: refused, and the handle stays usable."""
    torch, sysr, A, slab = system
    from emerge_gb300._lib import EmgError
    slab.factor(A, [0], precision)
    b = torch.ones((sysr.n, 2), dtype=torch.complex128, device="cuda")
    ref = slab.apply(b, [0, 0])
    torch.cuda.synchronize()
    with pytest.raises(EmgError):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            slab.apply(b, [0, 0])
    assert torch.equal(torch.view_as_real(slab.apply(b, [0, 0])), torch.view_as_real(ref))
