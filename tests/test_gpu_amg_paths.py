"""Which form of the multigrid CG a solve runs, by its launches: the one-launch form has
one per refinement beside the start, the refinements and the end, the separate
launches several per iteration.  The choice is made in every solve, so one handle
changes forms and smoothers.
"""

import pytest
import torch

from torchfem_gb300 import Planar, PlanarHeat, Solid, SolidHeat, _lib, mesh
from torchfem_gb300 import materials as M

pytestmark = pytest.mark.gpu

E3, E2 = M.IsotropicElasticity3D(1.0, 0.3), M.IsotropicElasticityPlaneStress(1.0, 0.3)
K3, K2 = M.IsotropicConductivity3D(1.0), M.IsotropicConductivity2D(1.0)
CASES = {
    "hexa": lambda: Solid(*mesh.cube_hexa(12, 11, 13), E3),
    "hexa-two-ctas": lambda: Solid(*mesh.cube_hexa(35, 32, 30), E3),
    "hexa-large": lambda: Solid(*mesh.cube_hexa(50, 50, 50), E3),  # beyond 64 MB a pass: always separate
    "quad": lambda: Planar(*mesh.rect_quad(60, 41), E2),
    "heat-quad": lambda: PlanarHeat(*mesh.rect_quad(50, 43), K2),
    "heat-hexa": lambda: SolidHeat(*mesh.cube_hexa(20, 21, 19), K3),
}


@pytest.mark.parametrize("name", CASES)
def test_form_of_every_solve(cuda, name):
    m = CASES[name]()
    m.constraints[m.nodes[:, 0] == 0.0] = True
    dm, lib = m.device_mesh, _lib.load()
    mesh_s, mat, refs = m._device_material()
    con = m.constraints.reshape(-1).to(cuda, torch.uint8).contiguous()
    b = torch.randn(dm.n_dofs, dtype=torch.float64, device=cuda, generator=torch.Generator(device=cuda).manual_seed(3))
    b[con.bool()] = 0.0
    s = dm.build_system(mesh_s, mat, con, "mixed", keep_refs=(refs,), precond="amg")
    try:
        for half, fused in ((1, 1), (0, 1), (1, 0), (0, 1), (1, 1), (0, 0), (1, 1)):
            lib.fem_amg_set_half_smoother(half)
            lib.fem_amg_set_fused_cycle(fused)
            before = lib.fem_launch_count()
            dm.solve(s, b, 1e-8, delta=1e-4)
            launches, st = lib.fem_launch_count() - before, s.stats
            assert st.iterations >= 4
            if fused and name != "hexa-large":
                # start 2, end 1; per refinement the iterations, the fold, the residual, the replacement
                assert launches <= 3 + 4 * (st.replacements + 1)
            else:
                assert launches >= 5 * st.iterations
    finally:
        lib.fem_amg_set_half_smoother(1)
        lib.fem_amg_set_fused_cycle(1)
