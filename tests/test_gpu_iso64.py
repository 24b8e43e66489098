"""FP64 element matrices of isotropic materials in moment form, at element
counts around the elements a CTA takes (one less, one more, a single element),
for every element type, against the general form.

Both sum at most eight points' products of a few FP64 factors: relative error
below 30 x 2^-53 of the summed magnitudes, which exceed the largest entry of an
element matrix by less than a factor of 20 on these meshes, so 1e-13 of that
entry.  The matrices are symmetric to the bit.
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


@pytest.mark.parametrize("n", [1, 3, 7, 8, 9, 15, 16, 17, 25])
@pytest.mark.parametrize("name", TYPES)
def test_moment_form_at_cta_remainders(cuda, name, n):
    model, (nodes, el), mat_ = TYPES[name]
    nodes = nodes + 0.02 * torch.rand(nodes.shape, generator=torch.Generator().manual_seed(n), dtype=torch.float64)
    el = el[:n]
    used, inv = torch.unique(el, return_inverse=True)
    m = model(nodes[used], inv.reshape(el.shape), mat_)
    assert len(m.elements) == n
    dm = m.device_mesh
    mesh_s, mat, _refs = m._device_material()
    assert mat.kind == _lib.FEM_MAT_ISO
    ref, k = dm.element_stiffness(mesh_s, mat), dm.element_stiffness64(mesh_s, mat)
    assert float((k - ref).abs().max()) <= 1e-13 * float(ref.abs().max())
    assert torch.equal(k, k.transpose(1, 2))
