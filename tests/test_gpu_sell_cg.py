"""The FP64 CG on the sliced block layout (FEM_FMT_SELL_F64) against the CSR
matrix that it is a copy of: the copy value by value, and the solution by its
residual in the CSR matrix, for every block size, for few slices and many
(four warps or one to a slice), slices with padding, a last slice of one row,
a node without elements, and the per-iteration kernels.

The systems are stiffness or conductivity matrices with twice their largest
diagonal entry m added to the diagonal: A >= 2 m I, and a row of at most 200
entries, none above m (3 m on the diagonal), gives ||A|| <= 202 m.  The
condition number is at most 101, so the recursive residual follows the true
one, and ||b - A x|| <= rtol ||b|| holds up to the rounding of A x, at most
200 * 2^-53 ||A|| ||x|| <= 200 * 1.1e-16 * 101 ||b|| < 1e-11 ||b||, with rtol =
1e-10.
"""

import ctypes as C

import pytest
import torch

from torchfem_gb300 import Planar, PlanarHeat, Solid, SolidHeat, _lib, mesh
from torchfem_gb300 import materials as M

pytestmark = pytest.mark.gpu

E3, E2 = M.IsotropicElasticity3D(1.0, 0.3), M.IsotropicElasticityPlaneStress(1.0, 0.3)
K3, K2 = M.IsotropicConductivity3D(1.0), M.IsotropicConductivity2D(1.0)


def _orphan(nodes, el):
    return torch.cat([nodes[:5], nodes.mean(0, keepdim=True), nodes[5:]]), torch.where(el >= 5, el + 1, el)


CASES = {
    "hexa-1-slice": lambda: Solid(*mesh.cube_hexa(2, 3, 4), E3),
    "hexa-99-rows": lambda: Solid(*mesh.cube_hexa(3, 11, 3), E3),
    "hexa-odd": lambda: Solid(*mesh.cube_hexa(12, 7, 9), E3),
    "hexa-many": lambda: Solid(*mesh.cube_hexa(49, 50, 51), E3),
    "tetra2-padded": lambda: Solid(*mesh.linear_to_quadratic(*mesh.box_tetra6(5, 4, 3)), E3),
    "tetra1-orphan": lambda: Solid(*_orphan(*mesh.cube_tetra(6, 5, 4)), E3),
    "quad-odd": lambda: Planar(*mesh.rect_quad(13, 29), E2),
    "quad-many": lambda: Planar(*mesh.rect_quad(160, 130), E2),
    "heat-odd": lambda: SolidHeat(*mesh.cube_hexa(8, 9, 10), K3),
    "heat-many": lambda: PlanarHeat(*mesh.rect_quad(150, 131), K2),
}


@pytest.mark.parametrize("name", CASES)
def test_sliced_cg_solves_the_csr_system(cuda, name, monkeypatch):
    m = CASES[name]()
    dm = m.device_mesh
    d = dm.d
    mesh_s, mat, refs = m._device_material()
    con = torch.zeros(dm.n_dofs, dtype=torch.uint8, device=cuda)
    val = dm.assemble_csr(dm.element_stiffness(mesh_s, mat), con)
    val[dm.diag_map] += 2.0 * val[dm.diag_map].max()
    A = torch.sparse_csr_tensor(dm.row_ptr, dm.col.to(torch.int64), val, (dm.n_dofs, dm.n_dofs))

    # the copy: every stored value at its slot, zeros elsewhere
    base, col, n_slots = dm.sell()
    sval = torch.full((n_slots * d * d,), float("nan"), dtype=torch.float64, device=cuda)
    assert dm.lib.fem_csr_to_sell64(C.byref(dm.blocks), dm.row_ptr.data_ptr(), val.data_ptr(), base.data_ptr(),
                                    sval.data_ptr(), dm.stream) == _lib.FEM_OK
    slot = torch.arange(n_slots, device=cuda)
    sl = torch.searchsorted(base, slot, right=True) - 1
    a = 32 * sl + (slot - base[sl]) % 32
    k = (slot - base[sl]) // 32
    comp = torch.arange(d * d, device=cuda)
    at = base[sl, None] * d * d + (k[:, None] * d * d + comp) * 32 + (slot - base[sl])[:, None] % 32
    vals = sval[at]
    keep = a < dm.n_nod
    deg = torch.zeros_like(a)
    deg[keep] = dm.nbr_ptr[a[keep] + 1] - dm.nbr_ptr[a[keep]]
    stored = keep & (k < deg)
    assert not vals[~stored].any() and not vals.isnan().any()
    r = a[stored, None] * d + comp // d
    c = col[stored].to(torch.int64)[:, None] * d + comp % d
    got = torch.sparse_coo_tensor(torch.stack([r.ravel(), c.ravel()]), vals[stored].ravel(), A.shape).coalesce()
    want = torch.sparse_coo_tensor(dm.glob_idx(), val, A.shape).coalesce()
    diff = (got - want).coalesce().values()
    assert not diff.any()

    gen = torch.Generator(device=cuda).manual_seed(1)
    b = torch.randn(dm.n_dofs, dtype=torch.float64, device=cuda, generator=gen)
    monkeypatch.setattr(dm, "CG_CLUSTER_NNZ", {1: 0, 2: 0, 3: 0})
    monkeypatch.setattr(dm, "CG_SELL_PAD", 100.0)
    before = dm.lib.fem_get_cg_path()
    try:
        for path in (1, 0):
            dm.lib.fem_set_cg_path(path)
            sysm = dm.csr_system(val, con)
            x = dm.solve(sysm, b, 1e-10)
            assert dm.cg_matrix(sysm).format == _lib.FEM_FMT_SELL_F64
            assert float((b - A @ x).norm() / b.norm()) <= 1.1e-10
            assert 0 < sysm.stats.iterations < 60
            with pytest.raises(RuntimeError):
                dm.solve(sysm, b, 1e-10, max_iter=2)
            assert not dm.solve(sysm, torch.zeros_like(b), 1e-10).any()
            bad = b.clone()
            bad[-1] = float("inf")
            with pytest.raises(_lib.FemError):
                dm.solve(sysm, bad, 1e-10)
    finally:
        dm.lib.fem_set_cg_path(before)
    del refs
