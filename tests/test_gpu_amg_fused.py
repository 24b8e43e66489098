"""The multigrid CG as one launch (k_amg_cg) against the separate launches it
replaces, for every block size: one slice of rows, a last slice of one row,
several levels, one and two CTAs per SM, the FP32 and the FP16 smoother, and
the iteration limit.

Both forms stop on the same FP64 residual, so the solution is checked by that
residual, formed here from the FP64 CSR matrix.  Its rounding against the
solver's own (sums of at most 200 terms of relative error 2^-53, ||A|| ||x|| <=
cond ||b||, cond < 1e5 for these meshes) is below 2e-9 of the 1e-6 asked for.
The two forms differ in the order of their sums only: iteration counts within
one of each other per refinement.
"""

import pytest
import torch

from torchfem_gb300 import Planar, PlanarHeat, Solid, SolidHeat, _lib, mesh
from torchfem_gb300 import materials as M

pytestmark = pytest.mark.gpu

E3, E2 = M.IsotropicElasticity3D(1.0, 0.3), M.IsotropicElasticityPlaneStress(1.0, 0.3)
K3, K2 = M.IsotropicConductivity3D(1.0), M.IsotropicConductivity2D(1.0)
CASES = {
    "hexa-27": lambda: Solid(*mesh.cube_hexa(3, 3, 3), E3),
    "hexa-33": lambda: Solid(*mesh.cube_hexa(11, 3, 1 + 1), E3),
    "hexa-levels": lambda: Solid(*mesh.cube_hexa(15, 14, 17), E3),
    "hexa-two-ctas": lambda: Solid(*mesh.cube_hexa(35, 32, 30), E3),
    "quad-66": lambda: Planar(*mesh.rect_quad(11, 6), E2),
    "quad-levels": lambda: Planar(*mesh.rect_quad(90, 71), E2),
    "heat-65": lambda: PlanarHeat(*mesh.rect_quad(13, 5), K2),
    "heat-levels": lambda: SolidHeat(*mesh.cube_hexa(30, 28, 27), K3),
}


@pytest.mark.parametrize("half", [1, 0])
@pytest.mark.parametrize("name", CASES)
def test_fused_cg_matches_separate_launches(cuda, name, half):
    m = CASES[name]()
    m.constraints[m.nodes[:, 0] == 0.0] = True
    dm, lib = m.device_mesh, _lib.load()
    mesh_s, mat, refs = m._device_material()
    con = m.constraints.reshape(-1).to(cuda, torch.uint8).contiguous()
    val = dm.assemble_csr(dm.element_stiffness(mesh_s, mat), con)
    A = torch.sparse_csr_tensor(dm.row_ptr, dm.col.to(torch.int64), val, (dm.n_dofs, dm.n_dofs))
    b = torch.randn(dm.n_dofs, dtype=torch.float64, device=cuda, generator=torch.Generator(device=cuda).manual_seed(3))
    b[con.bool()] = 0.0
    its = {}
    try:
        lib.fem_amg_set_half_smoother(half)
        for fused in (1, 0):
            lib.fem_amg_set_fused_cycle(fused)
            s = dm.build_system(mesh_s, mat, con, "mixed", keep_refs=(refs,), precond="amg")
            x = dm.solve(s, b, 1e-6, delta=1e-4)
            assert float((b - A @ x).norm() / b.norm()) <= 1.01e-6
            again = dm.solve(s, b, 1e-6, delta=1e-4)
            assert torch.equal(x, again)
            its[fused] = (s.stats.iterations, s.stats.replacements)
            with pytest.raises(RuntimeError):
                dm.solve(s, b, 1e-12, max_iter=2, delta=1e-4)
            assert s.stats.iterations == 2
    finally:
        lib.fem_amg_set_half_smoother(1)
        lib.fem_amg_set_fused_cycle(1)
    assert abs(its[1][0] - its[0][0]) <= max(its[0][1], its[1][1], 1)
