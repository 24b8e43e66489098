"""Sliced solves whose last slice holds one row, for every block size, and shares of
dot products that fill a finisher's threads once and one time more.  The node counts are
asserted, so that a name cannot drift from its case.
"""

import pytest
import torch

from torchfem_gb300 import Planar, PlanarHeat, Solid, SolidHeat, _lib, mesh
from torchfem_gb300 import materials as M

pytestmark = pytest.mark.gpu

E3, E2 = M.IsotropicElasticity3D(1.0, 0.3), M.IsotropicElasticityPlaneStress(1.0, 0.3)
K3, K2 = M.IsotropicConductivity3D(1.0), M.IsotropicConductivity2D(1.0)
ONE_ROW = {  # (nodes, model)
    "hexa": (225, lambda: Solid(*mesh.cube_hexa(3, 3, 25), E3)),
    "hexa-many": (35937, lambda: Solid(*mesh.cube_hexa(33, 33, 33), E3)),
    "quad": (33, lambda: Planar(*mesh.rect_quad(11, 3), E2)),
    "quad-many": (20769, lambda: Planar(*mesh.rect_quad(161, 129), E2)),
    "heat-quad": (65, lambda: PlanarHeat(*mesh.rect_quad(13, 5), K2)),
    "heat-hexa": (3969, lambda: SolidHeat(*mesh.cube_hexa(21, 21, 9), K3)),
}
SHARES = {  # (slices, model): a cluster of 8 x 256 threads adds 2,048 shares a round
    "2048": (2048, lambda: PlanarHeat(*mesh.rect_quad(257, 255), K2)),
    "2049": (2049, lambda: PlanarHeat(*mesh.rect_quad(331, 198), K2)),
}


def _system(m, cuda):
    m.constraints[m.nodes[:, 0] == 0.0] = True
    dm = m.device_mesh
    mesh_s, mat, refs = m._device_material()
    con = m.constraints.reshape(-1).to(cuda, torch.uint8).contiguous()
    val = dm.assemble_csr(dm.element_stiffness(mesh_s, mat), con)
    A = torch.sparse_csr_tensor(dm.row_ptr, dm.col.to(torch.int64), val, (dm.n_dofs, dm.n_dofs))
    b = torch.randn(dm.n_dofs, dtype=torch.float64, device=cuda, generator=torch.Generator(device=cuda).manual_seed(3))
    b[con.bool()] = 0.0
    return dm, (mesh_s, mat, con, refs), val, A, b


def _residual(A, x, b):
    return float((b - A @ x).norm() / b.norm())


@pytest.mark.parametrize("name", ONE_ROW)
def test_last_slice_of_one_row(cuda, name, monkeypatch):
    """FP64 CG on sliced blocks, and the multigrid CG in both forms, to 1e-6; the rounding
    of a residual is below 2e-9 of that (200 terms, ||A|| ||x|| <= 1e5 ||b||)."""
    nodes, make = ONE_ROW[name]
    m = make()
    assert len(m.nodes) == nodes and nodes % 32 == 1
    dm, (mesh_s, mat, con, refs), val, A, b = _system(m, cuda)
    monkeypatch.setattr(dm, "CG_CLUSTER_NNZ", {1: 0, 2: 0, 3: 0})
    monkeypatch.setattr(dm, "CG_SELL_PAD", 100.0)
    sysm = dm.csr_system(val, con)
    assert _residual(A, dm.solve(sysm, b, 1e-6), b) <= 1.01e-6
    assert dm.cg_matrix(sysm).format == _lib.FEM_FMT_SELL_F64
    lib = _lib.load()
    s = dm.build_system(mesh_s, mat, con, "mixed", keep_refs=(refs,), precond="amg")
    try:
        for half in (1, 0):
            for fused in (1, 0):
                lib.fem_amg_set_half_smoother(half)
                lib.fem_amg_set_fused_cycle(fused)
                assert _residual(A, dm.solve(s, b, 1e-6, delta=1e-4), b) <= 1.01e-6
    finally:
        lib.fem_amg_set_half_smoother(1)
        lib.fem_amg_set_fused_cycle(1)


@pytest.mark.parametrize("name", SHARES)
def test_rounds_of_shares(cuda, name):
    """A share left out of a second round would change alpha and beta: more iterations
    than the form that sums in another way, or a residual missed."""
    slices, make = SHARES[name]
    m = make()
    assert (len(m.nodes) + 31) // 32 == slices
    dm, (mesh_s, mat, con, refs), _, A, b = _system(m, cuda)
    lib = _lib.load()
    s = dm.build_system(mesh_s, mat, con, "mixed", keep_refs=(refs,), precond="amg")
    its = []
    try:
        for fused in (1, 0):
            lib.fem_amg_set_fused_cycle(fused)
            x = dm.solve(s, b, 1e-6, delta=1e-4)
            assert _residual(A, x, b) <= 1.01e-6
            assert torch.equal(x, dm.solve(s, b, 1e-6, delta=1e-4))
            its.append((s.stats.iterations, s.stats.replacements))
    finally:
        lib.fem_amg_set_fused_cycle(1)
    assert abs(its[0][0] - its[1][0]) <= max(its[0][1], its[1][1], 1)
