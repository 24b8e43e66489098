"""Element kernels with a form for small meshes and one for meshes that fill the GPU,
at the element counts where the dispatch changes.  The meshes are copies of a small
one, so that its results, checked elsewhere against autograd and the oracles, are the
reference: its own form, on the same numbers.
"""

import pytest
import torch

from torchfem_gb300 import Planar, mesh
from torchfem_gb300 import materials as M

pytestmark = pytest.mark.gpu

E2 = M.IsotropicElasticityPlaneStrain(1.0, 0.3)
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
