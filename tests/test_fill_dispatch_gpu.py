"""Fills at the sizes where their launches change (one launch for a small mesh, sliced element
blocks), real and complex mu, and rows next to an entity of the FP64 fill, against the oracle
within 1e-12 of each row's largest entry."""
import numpy as np
import pytest

import oracle
from _fixtures import rel_to_rowmax

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from emerge_gb300 import _build
    _build.build()
    return torch


def _materials(nT, seed, complex_mu):
    rng = np.random.default_rng(seed)
    eye = np.eye(3)[:, :, None]
    er = rng.uniform(1, 10, nT) * (1 - 1j * rng.uniform(0.001, 0.02, nT))
    ur = rng.uniform(0.5, 3, nT) + (0 if not complex_mu else -1j * rng.uniform(0.01, 0.1, nT))
    if complex_mu:
        ur[1:] = ur[1:].real                       # one lossy tet is enough for an imaginary part
    return eye * er[None, None], eye * (ur + 0j)[None, None]


# 4-7 cells: the one-launch fill ends at 155,648 positions (about 5.5 cells); 9-21 cells: ten, five,
# three and one slices of the element blocks (48, 120 and 240 CTAs of 128 tets)
@pytest.mark.parametrize("cells", [(1, 1, 1), (2, 3, 1), (5, 5, 5), (5, 5, 6), (6, 5, 6), (10, 10, 10), (12, 13, 12),
                                   (16, 17, 16), (18, 18, 18)])
@pytest.mark.parametrize("complex_mu", [False, True])
def test_boxes(torch_cuda, cells, complex_mu):
    from emerge_gb300.assembly import tet_mass_stiffness_matrices
    from emerge_gb300.mesh import Nedelec2Basis, structured_box
    m = structured_box(*(np.linspace(0.0, 1e-2 * n, n + 1) for n in cells), jitter=0.15, seed=3)
    field = Nedelec2Basis(m)
    er, ur = _materials(m.n_tets, sum(cells), complex_mu)
    E, B = tet_mass_stiffness_matrices(field, er, ur)
    Eo, Bo = oracle.tet_mass_stiffness_matrices(field, er, ur)
    assert np.array_equal(E.indptr, Eo.indptr) and np.array_equal(E.indices, Eo.indices)
    assert rel_to_rowmax(E, Eo) <= TOL and rel_to_rowmax(B, Bo) <= TOL
    assert complex_mu == bool(np.any(E.data.imag))


def test_materials_alternate_on_one_plan(torch_cuda):
    """Real, complex and real mu again on one plan: the flag of the complex fill does not stay."""
    torch = torch_cuda
    from emerge_gb300.assembly import AssemblyPlan, material_scalars
    from emerge_gb300.mesh import Nedelec2Basis, unit_cube
    for n in (4, 9):
        m = unit_cube(n, jitter=0.1, seed=2)
        plan = AssemblyPlan(Nedelec2Basis(m))
        outs = []
        for complex_mu in (False, True, False):
            eps, nu = material_scalars(*_materials(m.n_tets, 6, complex_mu))
            E, B = plan.assemble(torch.as_tensor(eps, device="cuda"), torch.as_tensor(nu, device="cuda"))
            outs.append((torch.view_as_real(E).clone(), torch.view_as_real(B).clone()))
        assert torch.equal(outs[0][0], outs[2][0]) and torch.equal(outs[0][1], outs[2][1])
        assert bool((outs[1][0][:, 1] != 0).any()) and not bool((outs[0][0][:, 1] != 0).any())


@pytest.mark.parametrize("complex_mu", [False, True])
@pytest.mark.parametrize("ring", [3, 12, 13, 20])
def test_fan(torch_cuda, ring, complex_mu):
    """One edge with ``ring`` tets: with more than twelve it leaves the fast fill, and the other
    entities' rows no longer follow each other."""
    from emerge_gb300.assembly import tet_mass_stiffness_matrices
    from emerge_gb300.mesh import Nedelec2Basis, TetMesh
    ang = 2 * np.pi * np.arange(ring) / ring
    pts = np.stack([np.cos(ang), np.sin(ang), 0.5 + 0.1 * np.sin(3 * ang)])
    nodes = np.concatenate([np.array([[0, 0], [0, 0], [0, 1.0]]), pts], axis=1)
    k = np.arange(ring)
    m = TetMesh(nodes, np.stack([0 * k, 0 * k + 1, 2 + k, 2 + (k + 1) % ring]))
    field = Nedelec2Basis(m)
    er, ur = _materials(ring, ring, complex_mu)
    E, B = tet_mass_stiffness_matrices(field, er, ur)
    Eo, Bo = oracle.tet_mass_stiffness_matrices(field, er, ur)
    assert rel_to_rowmax(E, Eo) <= TOL and rel_to_rowmax(B, Bo) <= TOL


@pytest.mark.parametrize("ring", [3, 6, 7, 12, 13])
def test_tensor_fan(torch_cuda, ring):
    """Full tensors around one edge: two edges or one to a group (six, seven tets), the largest
    group (twelve), and the FP64 fill next to the groups (thirteen)."""
    from emerge_gb300.assembly import tet_mass_stiffness_matrices
    from emerge_gb300.mesh import Nedelec2Basis, TetMesh
    ang = 2 * np.pi * np.arange(ring) / ring
    pts = np.stack([np.cos(ang), np.sin(ang), 0.5 + 0.1 * np.sin(3 * ang)])
    nodes = np.concatenate([np.array([[0, 0], [0, 0], [0, 1.0]]), pts], axis=1)
    k = np.arange(ring)
    m = TetMesh(nodes, np.stack([0 * k, 0 * k + 1, 2 + k, 2 + (k + 1) % ring]))
    field = Nedelec2Basis(m)
    rng = np.random.default_rng(ring)
    er, ur = (rng.uniform(-0.3, 0.3, (3, 3, ring)) + 1j * rng.uniform(-0.03, 0.03, (3, 3, ring)) for _ in range(2))
    er[range(3), range(3)] += 4.0
    ur[range(3), range(3)] += 1.5
    E, B = tet_mass_stiffness_matrices(field, er, ur)
    Eo, Bo = oracle.tet_mass_stiffness_matrices(field, er, ur)
    assert np.array_equal(E.indptr, Eo.indptr) and np.array_equal(E.indices, Eo.indices)
    assert rel_to_rowmax(E, Eo) <= TOL and rel_to_rowmax(B, Bo) <= TOL


def test_memory_of_a_plan(torch_cuda):
    """A plan keeps per tet its staged blocks (6400 B), invariants, scales, record and incidences, per matrix
    entry a column and half a descriptor, and own-column tables for edges alone."""
    torch = torch_cuda
    from emerge_gb300.assembly import AssemblyPlan
    from emerge_gb300.mesh import Nedelec2Basis, unit_cube
    m = unit_cube(40)
    field = Nedelec2Basis(m)
    AssemblyPlan(Nedelec2Basis(unit_cube(2)))      # the library and its tables are loaded
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    used = lambda: -torch.cuda.mem_get_info()[0] - torch.cuda.memory_reserved()  # noqa: E731
    before = used()
    plan = AssemblyPlan(field)
    torch.cuda.synchronize()
    N, nnz = int(field.n_field), int(plan.nnz)
    per_tet = 6400 + 344 + 32 + 16 + 544 + 80
    bound = per_tet * m.n_tets + 28 * N + (4 + 4) * nnz + 2 * m.n_edges * (12 * 4 + 4 * 16)
    assert used() - before <= bound + (64 << 20)   # 2 MB pages of some 25 arrays
