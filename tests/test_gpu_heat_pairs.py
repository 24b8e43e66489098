"""Conductivity matrices by node pairs at element counts around the elements a
CTA takes, for every element type, with symmetric and unsymmetric kappa and a
thickness, in FP64 and FP32, against einsum over the same gradients.

An entry sums at most 8 x 3 products of five FP64 factors: relative error below
40 x 2^-53 of the summed magnitudes, which exceed the largest entry by less than
a factor of 20 on these meshes, so 1e-13 of that entry; FP32 entries are the FP64
ones rounded (2^-24).
"""

import pytest
import torch

from torchfem_gb300 import PlanarHeat, SolidHeat, _lib, mesh
from torchfem_gb300 import materials as M

pytestmark = pytest.mark.gpu

K3, K2 = M.IsotropicConductivity3D(1.0), M.IsotropicConductivity2D(1.0)
HEXA, QUAD, TETRA = mesh.cube_hexa(4, 3, 6), mesh.rect_quad(8, 6), mesh.cube_tetra(3, 3, 3)
TRIA = QUAD[0], torch.cat([QUAD[1][:, [0, 1, 2]], QUAD[1][:, [0, 2, 3]]])
TYPES = {
    "hexa1": (SolidHeat, HEXA, K3), "hexa2": (SolidHeat, mesh.linear_to_quadratic(*HEXA), K3),
    "tetra1": (SolidHeat, TETRA, K3), "tetra2": (SolidHeat, mesh.linear_to_quadratic(*TETRA), K3),
    "quad1": (PlanarHeat, QUAD, K2), "quad2": (PlanarHeat, mesh.linear_to_quadratic(*QUAD), K2),
    "tria1": (PlanarHeat, TRIA, K2), "tria2": (PlanarHeat, mesh.linear_to_quadratic(*TRIA), K2),
}


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 17, 25])
@pytest.mark.parametrize("name", TYPES)
def test_pairs_at_cta_remainders(cuda, name, n, symmetric):
    model, (nodes, el), mat_ = TYPES[name]
    gen = torch.Generator().manual_seed(n)
    nodes = nodes + 0.02 * torch.rand(nodes.shape, generator=gen, dtype=torch.float64)
    used, inv = torch.unique(el[:n], return_inverse=True)
    m = model(nodes[used], inv.reshape(n, -1), mat_)
    dm = m.device_mesh
    _, mat, _refs = m._device_material()
    d = nodes.shape[1]
    kap = torch.eye(d, dtype=torch.float64) + 0.2 * torch.rand(n, d, d, generator=gen, dtype=torch.float64)
    if symmetric:
        kap = 0.5 * (kap + kap.transpose(1, 2))
    kap = kap.to(cuda).contiguous()
    th = 0.5 + torch.rand(n, generator=gen, dtype=torch.float64).to(cuda)
    mesh_s, own = dm.make_mesh(th), _lib.FemMaterial(mat.kind, kap.data_ptr())
    B = dm.bt.reshape(-1, n, el.shape[1], d)
    w = dm.weights.to(cuda)[:, None] * dm.detj.reshape(-1, n) * th
    ref = torch.einsum("pe,peai,eij,pebj->eab", w, B, kap, B)
    k = dm.element_stiffness(mesh_s, own)
    scale = float(ref.abs().max())
    assert float((k - ref).abs().max()) <= 1e-13 * scale
    assert not symmetric or torch.equal(k, k.transpose(1, 2))
    k32 = dm.element_stiffness(mesh_s, own, torch.float32)
    assert torch.equal(k32, k.float())


WANTED = ["want_sig", "want_mat", "want_thick", "want_de0", "want_v"]


@pytest.mark.parametrize("wants", [WANTED, [], *([w] for w in WANTED)])
@pytest.mark.parametrize("name", ["hexa1", "tetra2", "quad1"])
def test_reverse_of_fluxes(cuda, name, wants):
    """Every output alone and all at once, against autograd over the formula
    (the bound above; the reverse sums are as long)."""
    model, (nodes, el), mat_ = TYPES[name]
    gen = torch.Generator().manual_seed(4)
    m = model(nodes, el, mat_)
    dm, d, n = m.device_mesh, nodes.shape[1], len(el)
    _, mat, _refs = m._device_material()
    rnd = lambda *s: (torch.rand(s, generator=gen, dtype=torch.float64) - 0.3).to(cuda)  # noqa: E731
    B, conn = dm.bt.reshape(-1, n, el.shape[1], d), el.to(cuda)
    nip = B.shape[0]
    leaves = rnd(nip, n, d), rnd(n, d, d), 1.0 + rnd(n), rnd(n, d), rnd(dm.n_dofs)
    fp, kap, th, e0, v = (t.requires_grad_() for t in leaves)
    g, gflux, gh = rnd(dm.n_dofs), rnd(nip, n, d), rnd(nip, n, d)
    grad = torch.einsum("ea,peai->pei", v[conn], B)
    flux = fp + torch.einsum("eij,pej->pei", kap, grad - e0)
    w = dm.weights[:, None] * dm.detj.reshape(-1, n) * th
    f = torch.einsum("pe,peai,pei->ea", w, B, flux)
    refs = torch.autograd.grad((f * g[conn]).sum() + (flux * gflux).sum() + (grad * gh).sum(), (fp, kap, th, e0, v))
    keep = [t.detach().contiguous() for t in leaves]
    got = dm.vjp(dm.make_mesh(keep[2]), _lib.FemMaterial(mat.kind, keep[1].data_ptr()), keep[4], g,
                 sigma_prev=keep[0], de0=keep[3], gflux=gflux, gh=gh, mat_numel=kap.numel(),
                 **{k: True for k in wants})
    for k, a, ref in zip(WANTED, got, refs):
        assert (a is not None) == (k in wants)
        if a is not None:
            assert float((a.reshape(ref.shape) - ref).abs().max()) <= 1e-12 * float(ref.abs().max()), k
