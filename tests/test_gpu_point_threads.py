"""Element kernels with threads per point, per tangent entry and per node pair,
where their splits change: one element, elements around a CTA's, one element per
SM and one more, and meshes that fill CTAs.

Tangent stiffness, Neo-Hookean forces, tangents and reverse mode against the same
formulas in torch (autograd): sums of at most 8 x 27 products of a few FP64
factors, below 400 x 2^-53 of the summed magnitudes, which exceed the largest
result by less than a factor of 20 on these meshes: 1e-12 of it.  The FP32 form
likewise with 2^-24 and its rounded inputs: 2e-4.  J2 plasticity: an element's
results do not depend on the split, to the bit.
"""

import pytest
import torch

from torchfem_gb300 import Planar, Solid, _lib, mesh
from torchfem_gb300 import materials as M

pytestmark = pytest.mark.gpu

E3, E2 = M.IsotropicElasticity3D(1.0, 0.3), M.IsotropicElasticityPlaneStrain(1.0, 0.3)
HEXA, QUAD, TETRA = mesh.cube_hexa(4, 3, 6), mesh.rect_quad(8, 6), mesh.cube_tetra(3, 3, 3)
TRIA = QUAD[0], torch.cat([QUAD[1][:, [0, 1, 2]], QUAD[1][:, [0, 2, 3]]])
TYPES = {
    "hexa1": (Solid, HEXA, E3), "hexa2": (Solid, mesh.linear_to_quadratic(*HEXA), E3),
    "tetra1": (Solid, TETRA, E3), "tetra2": (Solid, mesh.linear_to_quadratic(*TETRA), E3),
    "quad1": (Planar, QUAD, E2), "quad2": (Planar, mesh.linear_to_quadratic(*QUAD), E2),
    "tria1": (Planar, TRIA, E2), "tria2": (Planar, mesh.linear_to_quadratic(*TRIA), E2),
}


def _model(model, nodes, el, mat, n, gen):
    nodes = nodes + 0.01 * torch.rand(nodes.shape, generator=gen, dtype=torch.float64) * (el.shape[0] < 100)
    used, inv = torch.unique(el[:n], return_inverse=True)
    m = model(nodes[used], inv.reshape(-1, el.shape[1]), mat)
    dm = m.device_mesh
    n = len(m.elements)
    B = dm.bt.reshape(-1, n, el.shape[1], nodes.shape[1])
    return m, dm, n, B, dm.weights[:, None] * dm.detj.reshape(-1, n)


def close(a, b, tol):
    return float((a.reshape(b.shape).double() - b).abs().max()) <= tol * float(b.abs().max())


@pytest.mark.parametrize("kind", [_lib.FEM_MAT_GENERAL, _lib.FEM_MAT_TANGENT_IP])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 16, 17, 25])
@pytest.mark.parametrize("name", TYPES)
def test_tangent_stiffness(cuda, name, n, kind):
    model, (nodes, el), mat_ = TYPES[name]
    gen = torch.Generator().manual_seed(n)
    _, dm, n, B, w = _model(model, nodes, el, mat_, n, gen)
    d, nip = nodes.shape[1], B.shape[0]
    C = torch.rand((nip if kind == _lib.FEM_MAT_TANGENT_IP else 1, n, d, d, d, d), generator=gen, dtype=torch.float64)
    C = C.to(cuda).contiguous()
    th = 0.5 + torch.rand(n, generator=gen, dtype=torch.float64).to(cuda)
    ref = torch.einsum("pe,peaj,peijkl,pebl->eaibk", w * th, B, C.expand(nip, -1, -1, -1, -1, -1), B)
    args = dm.make_mesh(th), _lib.FemMaterial(kind, C.data_ptr())
    assert close(dm.element_stiffness(*args), ref, 1e-12)
    assert close(dm.element_stiffness(*args, torch.float32), ref, 2e-4)


SOLIDS = {"hexa1": mesh.cube_hexa(18, 18, 18), "tetra1": mesh.cube_tetra(11, 11, 11),
          "tetra2": mesh.linear_to_quadratic(*mesh.cube_tetra(11, 11, 11))}


@pytest.mark.parametrize("n", [1, 152, 153, 4900])
@pytest.mark.parametrize("name", SOLIDS)
def test_neo_hookean(cuda, name, n):
    gen = torch.Generator().manual_seed(n)
    m, dm, n, B, w = _model(Solid, *SOLIDS[name], E3, n, gen)
    rnd = lambda *s: torch.rand(s, generator=gen, dtype=torch.float64).to(cuda)  # noqa: E731
    nip, conn = B.shape[0], m.elements.to(cuda)
    v = (0.002 * rnd(dm.n_dofs)).requires_grad_()
    params = (0.5 + rnd(n, 2)).requires_grad_()
    Fp = (torch.eye(3, dtype=torch.float64, device=cuda) + 0.05 * rnd(nip, n, 3, 3)).requires_grad_()
    F = Fp + torch.einsum("eac,peaj->pecj", v.reshape(-1, 3)[conn], B)
    J, Fi = torch.det(F), torch.linalg.inv(F)
    mu, lam = params[:, 0][None, :, None, None], params[:, 1][None, :, None, None]
    lnJ, Ft = torch.log(J)[..., None, None], Fi.transpose(-1, -2)
    P = mu * F + (lam * lnJ - mu) * Ft
    flux = F @ P / J[..., None, None]
    fe = torch.einsum("pe,peaj,pecj->eac", w, B, P)
    eye = torch.eye(3, dtype=torch.float64, device=cuda)
    m6, l6 = mu[..., None, None], lam[..., None, None]
    A = (m6 * torch.einsum("ik,JL->iJkL", eye, eye) + l6 * torch.einsum("peJi,peLk->peiJkL", Fi, Fi)
         + (m6 - l6 * lnJ[..., None, None]) * torch.einsum("peJk,peLi->peiJkL", Fi, Fi))
    mesh_s = dm.make_mesh(None)
    par, F0, vd = params.detach().contiguous(), Fp.detach().contiguous(), v.detach()
    out = dm.hyper_force(mesh_s, par, vd, F_prev=F0, want_tangent=True, want_flux=True, want_F=True, want_P=True)
    for got, ref in zip(out, (fe, A, flux, F, P)):
        assert close(got, ref.detach(), 1e-12)
    g, gflux, gF = rnd(dm.n_dofs) - 0.5, rnd(nip, n, 3, 3) - 0.5, rnd(nip, n, 3, 3) - 0.5
    loss = (fe * g.reshape(-1, 3)[conn]).sum() + (flux * gflux).sum() + (F * gF).sum()
    refs = torch.autograd.grad(loss, (Fp, params, v))
    got = dm.hyper_vjp(mesh_s, par, vd, g, F_prev=F0, gflux=gflux, gF=gF, want_Fprev=True, want_params=True,
                       want_v=True)
    for a, ref in zip(got, refs):
        assert close(a, ref, 1e-12)


@pytest.mark.parametrize("n", [1, 151, 153, 1217])
@pytest.mark.parametrize("quadratic", [False, True])
def test_plastic_split(cuda, quadratic, n):
    nodes, el = mesh.rect_quad(81, 81)
    if quadratic:
        nodes, el = mesh.linear_to_quadratic(nodes, el)
    gen = torch.Generator().manual_seed(n)
    u = 0.02 * torch.rand(nodes.shape, generator=gen, dtype=torch.float64)
    outs = []
    for k in (len(el), n):
        used, inv = torch.unique(el[:k], return_inverse=True)
        dm = Planar(nodes[used], inv.reshape(k, -1), E2).device_mesh
        params = torch.tensor([[1.0, 0.3, 0.01, 0.1]], dtype=torch.float64, device=cuda).repeat(k, 1)
        out = dm.plastic_force(dm.make_mesh(None), params, 1e-10, 10, u[used].reshape(-1).to(cuda),
                               want_tangent=True, want_outputs=True)
        outs.append([out[0].reshape(k, -1)[:n]] + [t.reshape(dm.nip, k, -1)[:, :n] for t in out[1:]])
    assert float(outs[0][3].abs().max()) > 0.0  # some points yield
    for a, b in zip(*outs):
        assert torch.equal(a, b)
