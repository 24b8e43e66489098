"""The dot products between the multigrid CG's separate launches
(k_dot_finish, k_cg_update), at row counts where the slices' shares fill one
thread, one CTA of the cluster, all of them, and more than one round of it.

A wrong or racing sum would change alpha or beta: CG then misses its 1e-6, two
solves differ, or it needs more iterations than the launch that sums another way.
The residual's own rounding is below 2e-9 of 1e-6 on these meshes (as for the
one-launch form).
"""

import pytest
import torch

from torchfem_gb300 import PlanarHeat, Solid, SolidHeat, _lib, mesh
from torchfem_gb300 import materials as M

pytestmark = pytest.mark.gpu

K3, K2 = M.IsotropicConductivity3D(1.0), M.IsotropicConductivity2D(1.0)
CASES = {
    "1-slice": lambda: PlanarHeat(*mesh.rect_quad(8, 4), K2),
    "255-slices": lambda: SolidHeat(*mesh.cube_hexa(24, 20, 17), K3),
    "257-slices": lambda: PlanarHeat(*mesh.rect_quad(257, 32), K2),
    "2049-slices": lambda: PlanarHeat(*mesh.rect_quad(257, 255), K2),
    "2250-slices": lambda: SolidHeat(*mesh.cube_hexa(50, 40, 36), K3),
    "blocks": lambda: Solid(*mesh.cube_hexa(41, 41, 41), M.IsotropicElasticity3D(1.0, 0.3)),
}


@pytest.mark.parametrize("name", CASES)
def test_separate_launch_dots(cuda, name):
    m = CASES[name]()
    m.constraints[m.nodes[:, 0] == 0.0] = True
    dm, lib = m.device_mesh, _lib.load()
    mesh_s, mat, refs = m._device_material()
    con = m.constraints.reshape(-1).to(cuda, torch.uint8).contiguous()
    A = dm.assemble_csr(dm.element_stiffness(mesh_s, mat), con)
    A = torch.sparse_csr_tensor(dm.row_ptr, dm.col.to(torch.int64), A, (dm.n_dofs, dm.n_dofs))
    b = torch.randn(dm.n_dofs, dtype=torch.float64, device=cuda, generator=torch.Generator(device=cuda).manual_seed(7))
    b[con.bool()] = 0.0
    s = dm.build_system(mesh_s, mat, con, "mixed", keep_refs=(refs,), precond="amg")
    its = {}
    try:
        for fused in (1, 0):
            lib.fem_amg_set_fused_cycle(fused)
            x = dm.solve(s, b, 1e-6, delta=1e-4)
            assert float((b - A @ x).norm() / b.norm()) <= 1.01e-6
            assert torch.equal(x, dm.solve(s, b, 1e-6, delta=1e-4))
            its[fused] = (s.stats.iterations, s.stats.replacements)
    finally:
        lib.fem_amg_set_fused_cycle(1)
    assert abs(its[1][0] - its[0][0]) <= max(its[0][1], its[1][1], 1)
