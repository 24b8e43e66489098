"""Element kernels with a form for small meshes and one for meshes that fill the GPU,
at the element counts where the dispatch changes.  The meshes are copies of a small
one, so that its results, checked elsewhere against autograd and the oracles, are the
reference: its own form, on the same numbers.
"""

import ctypes as C

import pytest
import torch

from torchfem_gb300 import Planar, PlanarHeat, Solid, SolidHeat, _lib, mesh
from torchfem_gb300 import materials as M

pytestmark = pytest.mark.gpu

E3, E2 = M.IsotropicElasticity3D(1.0, 0.3), M.IsotropicElasticityPlaneStrain(1.0, 0.3)
QUAD = mesh.rect_quad(5, 4)
TRIA = QUAD[0], torch.cat([QUAD[1][:, [0, 1, 2]], QUAD[1][:, [0, 2, 3]]])
PLANE = {"quad1": QUAD, "quad2": mesh.linear_to_quadratic(*QUAD), "tria1": TRIA,
         "tria2": mesh.linear_to_quadratic(*TRIA)}


def counts(wave, *at):
    """Element counts just below, at and just above multiples of a wave."""
    return sorted({int(wave * a) + k for a in at for k in (-1, 0, 1)})


def tile(t, n):
    """The first n rows of copies of t."""
    return t.repeat(-(-n // t.shape[0]), *[1] * (t.dim() - 1))[:n].contiguous()


def copies(nodes, el, n):
    """Nodes and the first n elements of copies of a mesh, and the number of copies."""
    c = -(-n // len(el))
    el = (el[None] + len(nodes) * torch.arange(c)[:, None, None]).reshape(-1, el.shape[1])[:n]
    return nodes.repeat(c, 1), el, c


def close(got, want, tol=1e-12):
    return float((got - want).abs().max()) <= tol * float(want.abs().max())


@pytest.fixture
def sms(cuda):
    return torch.cuda.get_device_properties(cuda).multi_processor_count


@pytest.mark.parametrize("name", PLANE)
def test_plastic_forms_agree(cuda, sms, name):
    """J2 forces, stresses, states and tangents: the same operations in both forms, which
    the compiler may contract differently, some 100 roundings of numbers at most ten
    times the largest result (the trial stress): 1e-12 of it."""
    gen = torch.Generator().manual_seed(5)
    nodes, el = PLANE[name]
    nodes = nodes + 0.02 * torch.rand(nodes.shape, generator=gen, dtype=torch.float64)
    k = len(el)
    u = 0.02 * torch.rand(nodes.shape, generator=gen, dtype=torch.float64)

    def run(n):
        big, elements, c = copies(nodes, el, n)
        dm = Planar(big, elements, E2).device_mesh
        v = u.repeat(c, 1).reshape(-1).to(cuda)
        one = torch.stack([1.0 + 0.1 * torch.arange(k), torch.full((k,), 0.3), torch.full((k,), 0.01),
                           torch.full((k,), 0.1)], 1).to(cuda, torch.float64)
        th = tile(0.5 + torch.arange(k, dtype=torch.float64, device=cuda) / k, n)
        out = dm.plastic_force(dm.make_mesh(th), tile(one, n), 1e-10, 10, v, want_tangent=True,
                               want_outputs=True)
        force = dm.plastic_force(dm.make_mesh(th), tile(one, n), 1e-10, 10, v)[0]
        dm.check_status("plastic")
        assert close(force, out[0])
        return [out[0].reshape(1, n, -1)] + [t.reshape(dm.nip, n, -1) for t in out[1:]]

    ref = run(k)
    assert float(ref[3].abs().max()) > 0.0  # some points yield
    per_sm = 64 if name == "tria1" else 128
    for n in counts(per_sm * sms, 1.0) if name == "tria1" else counts(per_sm * sms, 4 / 5, 1.0, 2 * 4 / 5, 4.0):
        for got, want in zip(run(n), ref):
            assert close(got, want.repeat(1, -(-n // k), 1)[:, :n]), n


def test_single_point_neo_hookean(cuda, sms):
    """Linear tetrahedra: forces, tangents, fluxes and the reverse mode, some 200
    roundings of numbers at most ten times the largest result: 1e-12 of it."""
    gen = torch.Generator().manual_seed(6)
    nodes, el = mesh.cube_tetra(3, 3, 3)
    nodes = nodes + 0.02 * torch.rand(nodes.shape, generator=gen, dtype=torch.float64)
    k = len(el)
    rnd = lambda *s: torch.rand(s, generator=gen, dtype=torch.float64).to(cuda)  # noqa: E731
    u, g = 0.002 * rnd(len(nodes), 3), rnd(len(nodes), 3) - 0.5
    par, F0 = 0.5 + rnd(k, 2), torch.eye(3, dtype=torch.float64, device=cuda) + 0.05 * rnd(k, 3, 3)
    gflux, gF = rnd(k, 3, 3) - 0.5, rnd(k, 3, 3) - 0.5

    def run(n):
        big, elements, c = copies(nodes, el, n)
        m = Solid(big, elements, E3)
        dm = m.device_mesh
        ms, v, Fp, p = dm.make_mesh(None), u.repeat(c, 1).reshape(-1), tile(F0, n), tile(par, n)
        out = dm.hyper_force(ms, p, v, F_prev=Fp, want_tangent=True, want_flux=True, want_F=True, want_P=True)
        force = dm.hyper_force(ms, p, v, F_prev=Fp)[0]
        dm.check_status("hyper")
        assert close(force, out[0])
        back = dm.hyper_vjp(ms, p, v, g.repeat(c, 1).reshape(-1), F_prev=Fp, gflux=tile(gflux, n), gF=tile(gF, n),
                            want_Fprev=True, want_params=True)
        return [t.reshape(n, -1) for t in (*out, *back[:2])] + [hyper_v(dm, ms, p, v, g, Fp, c, n)]

    def hyper_v(dm, ms, p, v, g, Fp, c, n):
        """The element sums of the nodal cotangents, before they meet at a node."""
        gve = torch.full((n, 12), float("nan"), dtype=torch.float64, device=cuda)
        gn = g.repeat(c, 1).reshape(-1).contiguous()
        _lib.check(dm.lib.fem_hyper_vjp(C.byref(ms), p.data_ptr(), v.data_ptr(), None, None, 0, Fp.data_ptr(),
                                        gn.data_ptr(), None, None, None, None, gve.data_ptr(), dm.stream), "vjp")
        return gve

    ref = run(k)
    for n in counts(sms, 64, 512):
        for got, want in zip(run(n), ref):
            assert close(got, tile(want, n)), n


@pytest.mark.parametrize("name", ["tetra1", "tria1"])
def test_single_point_tangent_matrices(cuda, sms, name):
    """FP64 and FP32 matrices of unsymmetric tangents, per element and per point: sums of
    at most 9 products of a few factors, 40 x 2^-53 (2^-24) of the summed magnitudes, below
    20 times the largest entry: 1e-13 and 1e-4 of it."""
    gen = torch.Generator().manual_seed(7)
    solid = name == "tetra1"
    nodes, el = mesh.cube_tetra(3, 3, 3) if solid else TRIA
    nodes = nodes + 0.02 * torch.rand(nodes.shape, generator=gen, dtype=torch.float64)
    k, d = len(el), nodes.shape[1]
    tangent = torch.rand(k, d**4, generator=gen, dtype=torch.float64).to(cuda)
    th = 0.5 + torch.rand(k, generator=gen, dtype=torch.float64).to(cuda)

    def run(n, kind, dtype):
        big, elements, _ = copies(nodes, el, n)
        dm = (Solid if solid else Planar)(big, elements, E3 if solid else E2).device_mesh
        c, t = tile(tangent, n), tile(th, n)
        return dm.element_stiffness(dm.make_mesh(t), _lib.FemMaterial(kind, c.data_ptr()), dtype)

    for dtype, per_sm, tol in ((torch.float64, 192, 1e-13), (torch.float32, 1024, 1e-4)):
        for kind in (_lib.FEM_MAT_GENERAL, _lib.FEM_MAT_TANGENT_IP):
            ref = run(k, kind, dtype)
            for n in counts(sms, per_sm):
                assert close(run(n, kind, dtype), tile(ref, n), tol), n


@pytest.mark.parametrize("name", ["hexa1", "tetra1", "tetra2", "quad1", "quad2", "tria1", "tria2"])
def test_symmetric_conductivity_beside_another(cuda, name):
    """An element's conductivity matrix is the same to the bit whatever its neighbours'
    kappa, and symmetric where its own is."""
    solid = name[:2] in ("he", "te")
    grid = {"hexa": mesh.cube_hexa(4, 4, 6), "tetr": mesh.cube_tetra(3, 3, 4), "quad": QUAD, "tria": TRIA}[name[:4]]
    nodes, el = mesh.linear_to_quadratic(*grid) if name[-1] == "2" else grid
    gen = torch.Generator().manual_seed(8)
    nodes = nodes + 0.02 * torch.rand(nodes.shape, generator=gen, dtype=torch.float64)
    n, d = len(el), nodes.shape[1]
    m = (SolidHeat if solid else PlanarHeat)(nodes, el, (M.IsotropicConductivity3D if solid else
                                                         M.IsotropicConductivity2D)(1.0))
    dm = m.device_mesh
    _, mat, _refs = m._device_material()
    kap = torch.eye(d, dtype=torch.float64) + 0.2 * torch.rand(n, d, d, generator=gen, dtype=torch.float64)
    sym = (0.5 * (kap + kap.transpose(1, 2))).to(cuda).contiguous()
    odd = torch.arange(n) % 7 == 3
    mixed = torch.where(odd[:, None, None].to(cuda), kap.to(cuda), sym).contiguous()
    k_sym, k_mixed = (dm.element_stiffness(dm.make_mesh(None), _lib.FemMaterial(mat.kind, k.data_ptr()))
                      for k in (sym, mixed))
    even = ~odd.to(cuda)
    assert torch.equal(k_sym, k_sym.transpose(1, 2)) and torch.equal(k_sym[even], k_mixed[even])
    B = dm.bt.reshape(-1, n, el.shape[1], d)
    ref = torch.einsum("pe,peai,eij,pebj->eab", dm.weights[:, None] * dm.detj.reshape(-1, n), B, mixed, B)
    assert close(k_mixed, ref, 1e-13)  # the bound of the conductivity tests


@pytest.mark.parametrize("name", ["hexa1", "tetra1", "tetra2", "quad2", "tria1"])
def test_moment_form_of_few_and_many(cuda, sms, name):
    """Isotropic FP64 matrices where small CTAs end: the same sums, so the same to the
    bit, and against the general form within its bound."""
    solid = name[:2] in ("he", "te")
    nodes, el = {"hexa1": mesh.cube_hexa(4, 3, 3), "tetra1": mesh.cube_tetra(3, 3, 2),
                 "tetra2": mesh.linear_to_quadratic(*mesh.cube_tetra(2, 3, 2)),
                 "quad2": mesh.linear_to_quadratic(*QUAD), "tria1": TRIA}[name]
    nodes = nodes + 0.02 * torch.rand(nodes.shape, generator=torch.Generator().manual_seed(9), dtype=torch.float64)
    k = len(el)
    E = 1.0 + torch.arange(k, dtype=torch.float64) / k

    def run(n):
        big, elements, _ = copies(nodes, el, n)
        mat = (M.IsotropicElasticity3D if solid else M.IsotropicElasticityPlaneStrain)(tile(E, n), torch.tensor(0.3))
        m = (Solid if solid else Planar)(big, elements, mat)
        mesh_s, mat, _refs = m._device_material()
        dm = m.device_mesh
        return dm.element_stiffness_iso64(mesh_s, mat), dm.element_stiffness(mesh_s, mat)

    ref, general = run(k)
    assert close(ref, general, 1e-13)
    for n in counts(sms, 64 if name in ("tetra1", "tria1") else 4):
        assert torch.equal(run(n)[0], tile(ref, n)), n
