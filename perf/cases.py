"""Performance cases of the forward solve and its adjoint.

Each case is one finite-element analysis as a program that uses the package
runs it, through the public model classes: set the load and the material,
`solve(...)`, then the gradient of a scalar with respect to the inputs that
such a program differentiates (nodal forces, element moduli, densities,
thicknesses, conductivities).  Sizes are those of the repository's own
configurations (10^3 and 70^3 Hexa1 cubes, the 400 x 200 SIMP cantilever, the
Neo-Hookean Tetra2 box, the J2 O-grid plate, the thermal slab, the cylindrical
shell roof) and odd-sized generic ones between them.

Tolerances are the package's defaults or tighter: `stol` 1e-12 for the FP64
solver (the accuracy the tests ask of it) and 1e-10 for the mixed one (its
documented target).
"""

from __future__ import annotations

import itertools
import math
import sys
from pathlib import Path

import torch

_ROOT = Path(__file__).resolve().parent.parent
for _p in (_ROOT, _ROOT / "torch-fem_gb300"):
    if str(_p) not in sys.path:
        sys.path.insert(0, str(_p))

F64 = torch.float64
NU = torch.tensor(0.3, dtype=F64)


# ------------------------------------------------------------------- cases --
def listed():
    return [
        # smallest call: one load case on a part of a few thousand unknowns
        # (configuration 1), default FP64 solver; latency and launches count
        {"name": "box 10 fp64", "kind": "box", "nx": 10, "ny": 10, "nz": 10, "precision": "fp64", "wrt": "E"},
        # ordinary static analysis with the default solver, odd sizes
        {"name": "box 33x29x37 fp64", "kind": "box", "nx": 33, "ny": 29, "nz": 37, "precision": "fp64", "wrt": "E"},
        # large analysis with the default solver: the matrix leaves the L2 cache
        {"name": "box 52x47x50 fp64", "kind": "box", "nx": 52, "ny": 47, "nz": 50, "precision": "fp64", "wrt": "forces"},
        # the headline workload (configuration 2): 1.07M unknowns, mixed precision
        {"name": "box 70 mixed", "kind": "box", "nx": 70, "ny": 70, "nz": 70, "precision": "mixed", "wrt": "forces"},
        # a single analysis of a mesh that was not seen before: the model, its
        # pattern and the multigrid hierarchy are built inside the pass
        {"name": "new box 27x22x31 mixed", "kind": "new box", "nx": 27, "ny": 22, "nz": 31, "precision": "mixed",
         "wrt": "E"},
        # one step of a density optimisation on a small plane-stress design, default solver
        {"name": "simp 97x51 fp64", "kind": "simp", "nx": 97, "ny": 51, "precision": "fp64"},
        # the same at configuration 3's size, mixed precision
        {"name": "simp 400x200 mixed", "kind": "simp", "nx": 400, "ny": 200, "precision": "mixed"},
        # finite-strain Neo-Hookean pull on quadratic tetrahedra (configuration 4's
        # problem, reduced): many Newton corrections of one small system
        {"name": "hyper 6x2x2 fp64", "kind": "hyper", "nx": 6, "ny": 2, "nz": 2},
        # elasto-plastic plate with a hole (configuration 5's problem, reduced)
        {"name": "plate 32x8 fp64", "kind": "plate", "n_theta": 32, "n_rad": 8},
        # Tria1 shell roof: six unknowns per node, default solver
        {"name": "roof 33x27 fp64", "kind": "roof", "n_arc": 33, "n_len": 27},
        # steady heat conduction, the thermal benchmark's slab at its 1M-unknown
        # size with a random density field: one step of a thermal optimisation
        {"name": "slab 1024 mixed", "kind": "slab", "n": 1024},
        # transient heat conduction with gradients through all time steps
        {"name": "transient 101x89 fp64", "kind": "transient", "nx": 101, "ny": 89, "steps": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "box", "new box", "simp", "simp", "hyper", "plate", "roof", "slab", "transient"])
    if kind == "box":
        precision = rng.choice(["fp64", "mixed"])
        top = 46 if precision == "fp64" else 64
        n = _log_int(rng, 7, top)
        return {"kind": kind, "nx": n, "ny": max(5, n + rng.randint(-4, 4)), "nz": max(5, n + rng.randint(-4, 4)),
                "precision": precision, "wrt": rng.choice(["E", "forces"])}
    if kind == "new box":
        n = _log_int(rng, 9, 40)
        return {"kind": kind, "nx": n, "ny": max(7, n + rng.randint(-5, 5)), "nz": max(7, n + rng.randint(-5, 5)),
                "precision": "mixed", "wrt": "E"}
    if kind == "simp":
        precision = rng.choice(["fp64", "mixed"])
        nx = _log_int(rng, 30, 120) if precision == "fp64" else _log_int(rng, 60, 400)
        return {"kind": kind, "nx": nx, "ny": max(15, nx // 2 + rng.randint(-5, 0)), "precision": precision}
    if kind == "hyper":
        return {"kind": kind, "nx": rng.randint(5, 9), "ny": 2, "nz": rng.randint(2, 3)}
    if kind == "plate":
        return {"kind": kind, "n_theta": 8 * rng.randint(2, 4), "n_rad": rng.randint(5, 8)}
    if kind == "roof":
        return {"kind": kind, "n_arc": rng.randint(9, 41), "n_len": rng.randint(7, 33)}
    if kind == "slab":
        return {"kind": kind, "n": 2 * _log_int(rng, 40, 500)}
    return {"kind": kind, "nx": rng.randint(20, 120), "ny": rng.randint(20, 120), "steps": rng.randint(4, 12)}


# ------------------------------------------------------------------ inputs --
def _hexa_grid(nx, ny, nz, lx, ly, lz):
    """Nodes and Hexa1 elements of a structured box, x-major numbering."""
    x, y, z = torch.meshgrid(torch.linspace(0, lx, nx + 1, dtype=F64), torch.linspace(0, ly, ny + 1, dtype=F64),
                             torch.linspace(0, lz, nz + 1, dtype=F64), indexing="ij")
    ids = torch.arange((nx + 1) * (ny + 1) * (nz + 1)).reshape(nx + 1, ny + 1, nz + 1)
    corner = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
    el = torch.stack([ids[i:nx + i, j:ny + j, k:nz + k].ravel() for i, j, k in corner], dim=1)
    return torch.stack([x.ravel(), y.ravel(), z.ravel()], dim=1), el


def _quad_grid(nx, ny, lx, ly):
    x, y = torch.meshgrid(torch.linspace(0, lx, nx + 1, dtype=F64), torch.linspace(0, ly, ny + 1, dtype=F64),
                          indexing="ij")
    ids = torch.arange((nx + 1) * (ny + 1)).reshape(nx + 1, ny + 1)
    el = torch.stack([ids[i:nx + i, j:ny + j].ravel() for i, j in ((0, 0), (1, 0), (1, 1), (0, 1))], dim=1)
    return torch.stack([x.ravel(), y.ravel()], dim=1), el


def _inputs(case, seed):
    """Mesh, loads and fields of a case, from the seed alone."""
    gen = torch.Generator().manual_seed(seed)
    kind = case["kind"]
    if kind in ("box", "new box"):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        h = 1.0 / max(nx, ny, nz)
        nodes, el = _hexa_grid(nx, ny, nz, nx * h, ny * h, nz * h)
        hi = nodes.max(0).values
        inner = ((nodes > 0) & (nodes < hi)).all(1)
        nodes = nodes + inner[:, None] * (torch.rand(nodes.shape, generator=gen, dtype=F64) - 0.5) * (0.2 * h)
        E = 1000.0 * (1.0 + 0.1 * torch.randn(len(el), generator=gen, dtype=F64).clamp(-4, 4))
        x0, x1 = nodes[:, 0] == 0.0, nodes[:, 0] == hi[0]
        forces = torch.zeros_like(nodes)
        pull = torch.tensor([0.3, -0.2, -1.0], dtype=F64) + 0.2 * torch.randn(3, generator=gen, dtype=F64)
        noise = 1.0 + 0.2 * torch.rand(len(nodes), 1, generator=gen, dtype=F64)
        forces[x1] = (pull * noise / int(x1.sum()))[x1]
        d = {"nodes": nodes, "el": el, "E": E, "con": x0[:, None].expand(-1, 3).contiguous(), "forces": forces}
    elif kind == "simp":
        nx, ny = case["nx"], case["ny"]
        nodes, el = _quad_grid(nx, ny, nx / ny, 1.0)
        rho = 0.2 + 0.8 * torch.rand(len(el), generator=gen, dtype=F64)
        forces = torch.zeros_like(nodes)
        tip = int(((nodes - torch.tensor([nx / ny, 0.5], dtype=F64)) ** 2).sum(1).argmin())
        forces[tip, 1] = -1.0
        d = {"nodes": nodes, "el": el, "rho": rho, "con": (nodes[:, :1] == 0.0).expand(-1, 2).contiguous(),
             "forces": forces}
    elif kind == "hyper":
        from torchfem_gb300 import mesh

        nodes, el = mesh.linear_to_quadratic(*mesh.box_tetra6(case["nx"] + 1, case["ny"] + 1, case["nz"] + 1,
                                                              3.0, 1.0, 1.0))
        E = 1000.0 * (1.0 + 0.1 * torch.randn(len(el), generator=gen, dtype=F64))
        d = {"nodes": nodes, "el": el, "E": E}
    elif kind == "plate":
        from torchfem_gb300 import mesh

        nodes, el = mesh.plate_hole_ogrid(case["n_theta"], case["n_rad"])
        d = {"nodes": nodes, "el": el, "t": 1.0 + 0.1 * torch.rand(len(el), generator=gen, dtype=F64)}
    elif kind == "roof":
        from torchfem_gb300 import mesh

        nodes, el = mesh.cylinder_patch_tria(case["n_arc"], case["n_len"], 1.0, 2.0, 80.0)
        d = {"nodes": nodes, "el": el, "E": 1000.0 * (1.0 + 0.1 * torch.randn(len(el), generator=gen, dtype=F64)),
             "t": 0.05 * (1.0 + 0.2 * torch.rand(len(el), generator=gen, dtype=F64))}
    elif kind == "slab":
        n = case["n"]
        lz = 2.0 / n
        nodes, el = _hexa_grid(n, n // 2, 1, 2.0, 1.0, lz)
        right = nodes[:, 0] == 2.0
        wy = torch.full((len(nodes),), 1.0 / (n // 2), dtype=F64)
        wy[(nodes[:, 1] == 0.0) | (nodes[:, 1] == 1.0)] /= 2.0
        q = torch.zeros(len(nodes), 1, dtype=F64)
        q[right, 0] = wy[right] * (0.5 * lz)
        d = {"nodes": nodes, "el": el, "q": q, "con": nodes[:, :1] == 0.0,
             "rho": 0.4 + 0.2 * torch.rand(len(el), generator=gen, dtype=F64)}
    else:  # transient
        nodes, el = _quad_grid(case["nx"], case["ny"], 1.0, 1.0)
        kappa = 400.0 * (0.5 + torch.rand(len(el), generator=gen, dtype=F64))
        con = (nodes[:, :1] == 0.0) | (nodes[:, :1] == 1.0)
        temp = torch.zeros(len(nodes), 1, dtype=F64)
        temp[nodes[:, 0] == 0.0] = 5.0
        temp[nodes[:, 0] == 1.0] = 20.0
        d = {"nodes": nodes, "el": el, "kappa": kappa, "con": con, "temp": temp}
    # the shell model takes its tensors on the host
    return d if kind == "roof" else {k: v.to("cuda") for k, v in d.items()}


# ------------------------------------------------------------ prepare, run --
def _box_model(d):
    from torchfem_gb300 import Solid
    from torchfem_gb300.materials import IsotropicElasticity3D

    m = Solid(d["nodes"], d["el"], IsotropicElasticity3D(d["E"], NU))
    m.constraints = d["con"]
    m.forces = d["forces"]
    return m


def prepare(case, seed):
    from torchfem_gb300 import Planar, PlanarHeat, Shell, Solid, SolidHeat
    from torchfem_gb300 import materials as M

    d = _inputs(case, seed)
    kind = case["kind"]
    s = {"case": case, "d": d}
    if kind == "box":
        s["model"] = _box_model(d)
    elif kind == "simp":
        m = Planar(d["nodes"], d["el"], M.IsotropicElasticityPlaneStress(d["rho"] ** 3, NU))
        m.constraints = d["con"]
        m.forces = d["forces"]
        s["model"] = m
    elif kind == "hyper":
        m = Solid(d["nodes"], d["el"], None)
        right = d["nodes"][:, 0] == 3.0
        m.constraints[d["nodes"][:, 0] == 0.0, :] = True
        m.constraints[right, 0] = True
        m.displacements[right, 0] = 0.5
        s.update(model=m, right=right)
    elif kind == "plate":
        mat = M.IsotropicPlasticityPlaneStrain(torch.tensor(1000.0, dtype=F64), NU, lambda q: 1.0 + 100.0 * q,
                                               lambda q: 100.0 * torch.ones_like(q))
        nodes = d["nodes"]
        m = Planar(nodes, d["el"], mat, thickness=d["t"])
        left = torch.isclose(nodes[:, 0], torch.zeros_like(nodes[:, 0]))
        right = torch.isclose(nodes[:, 0], torch.full_like(nodes[:, 0], 2.0))
        pin = int(((nodes - torch.tensor([0.0, 0.5], dtype=F64, device=nodes.device)) ** 2).sum(1).argmin())
        m.constraints[left, 0] = True
        m.constraints[pin, 1] = True
        m.constraints[right, 0] = True
        m.displacements[right, 0] = 0.02
        s.update(model=m, right=right)
    elif kind == "roof":
        nodes = d["nodes"]
        m = Shell(nodes, d["el"], M.IsotropicElasticityPlaneStress(d["E"], NU), thickness=d["t"])
        y0, y1 = nodes[:, 1] == 0.0, nodes[:, 1] == 2.0
        side = (nodes[:, 0] - nodes[:, 0].min()).abs() < 1e-12
        m.constraints[y0, :] = True
        m.constraints[y1, :3] = True
        m.displacements[y1, 1] = 1e-3
        m.forces[:, 2] = -1.0 / len(nodes)
        m.forces[side, 3] = 2e-3
        s["model"] = m
    elif kind == "slab":
        m = SolidHeat(d["nodes"], d["el"], M.IsotropicConductivity3D(1.0))
        m.constraints = d["con"]
        m.heat_flux = d["q"]
        s["model"] = m
    elif kind == "transient":
        m = PlanarHeat(d["nodes"], d["el"], M.IsotropicConductivity2D(d["kappa"], 1.0e5))
        m.constraints = d["con"]
        m.temperatures = d["temp"]
        s["model"] = m
    return s


def run(state):
    from torchfem_gb300 import materials as M

    case, d = state["case"], state["d"]
    kind = case["kind"]
    if kind in ("box", "new box"):
        m = state["model"] if kind == "box" else _box_model(d)
        tol = {"stol": 1e-12 if case["precision"] == "fp64" else 1e-10, "precision": case["precision"]}
        if case["wrt"] == "forces":  # the adjoint field of the summed displacements
            p = d["forces"].detach().requires_grad_(True)
            m.forces = p
            u, f, s, F, _ = m.solve(differentiable_parameters=p, **tol)
            (g,) = torch.autograd.grad(u.sum(), p)
        else:  # compliance with respect to the element moduli
            p = d["E"].detach().requires_grad_(True)
            m.material = M.IsotropicElasticity3D(p, NU)
            u, f, s, F, _ = m.solve(differentiable_parameters=p, **tol)
            (g,) = torch.autograd.grad(torch.inner(d["forces"].ravel(), u.ravel()), p)
        return {"u": u, "f": f, "s": s, "F": F, "g": g}
    m = state.get("model")
    if kind == "simp":
        rho = d["rho"].detach().requires_grad_(True)
        m.material = M.IsotropicElasticityPlaneStress(rho**3, NU)
        u, f, s, F, _ = m.solve(stol=1e-12 if case["precision"] == "fp64" else 1e-10, precision=case["precision"],
                                differentiable_parameters=rho)
        (g,) = torch.autograd.grad(torch.inner(f.ravel(), u.ravel()), rho)
        return {"u": u, "f": f, "s": s, "F": F, "g": g}
    if kind == "hyper":
        E, nu = d["E"].detach().requires_grad_(True), 0.45
        mu, lbd = E / (2.0 * (1.0 + nu)), E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu))
        m.material = M.Hyperelastic3D(M.neo_hookean_psi, torch.stack([mu, lbd], -1))
        u, f, s, F, _ = m.solve(increments=torch.linspace(0.0, 1.0, 11, dtype=F64), nlgeom=True, rtol=1e-10, atol=1e-10,
                                max_iter=20, stol=1e-12, differentiable_parameters=E)
        (g,) = torch.autograd.grad(f[state["right"], 0].sum(), E)
        return {"u": u, "f": f, "s": s, "F": F, "g": g}
    if kind == "plate":
        t = d["t"].detach().requires_grad_(True)
        m.thickness = t
        u, f, s, F, q = m.solve(increments=torch.linspace(0.0, 1.0, 6, dtype=F64), rtol=1e-12, atol=1e-12, max_iter=80,
                                stol=1e-12, differentiable_parameters=t)
        (g,) = torch.autograd.grad(f[state["right"], 0].sum(), t)
        return {"u": u, "f": f, "s": s, "F": F, "q": q, "g": g}
    if kind == "roof":
        # membrane and bending moduli vary, the transverse shear moduli stay the model's
        E, t = d["E"].detach().requires_grad_(True), d["t"].detach().requires_grad_(True)
        m.material = M.IsotropicElasticityPlaneStress(E, NU)
        m.thickness = t
        u, f, s, _, _ = m.solve(stol=1e-12, rtol=1e-12, atol=1e-14, differentiable_parameters=(E, t))
        gE, gt = torch.autograd.grad(u.pow(2).sum(), (E, t))
        return {"u": u, "f": f, "s": s, "gE": gE, "gt": gt}
    if kind == "slab":
        rho = d["rho"].detach().requires_grad_(True)
        m.material = M.IsotropicConductivity3D(1e-3 + (1.0 - 1e-3) * rho**3)
        T, f, q, grad, _ = m.solve(stol=1e-10, precision="mixed", differentiable_parameters=rho)
        (g,) = torch.autograd.grad(torch.inner(d["q"].ravel(), T.ravel()), rho)
        return {"T": T, "f": f, "q": q, "grad": grad, "g": g}
    kappa = d["kappa"].detach().requires_grad_(True)
    m.material = M.IsotropicConductivity2D(kappa, 1.0e5)
    times = torch.linspace(0.0, 1.0 * case["steps"], case["steps"] // 2 + 1, dtype=F64)
    T, f, q, _, _ = m.time_integration(times, delta_t=1.0, stol=1e-12, rtol=1e-10, differentiable_parameters=kappa)
    (g,) = torch.autograd.grad(T[-1].pow(2).mean(), kappa)
    return {"T": T, "f": f, "q": q, "g": g}


# -------------------------------------------------------------------- work --
def work(case):
    """What one pass cannot do without: the mesh, the fields and the loads read
    once, every output written once; the element matrices of each step (the
    symmetric half) and one product with them per linear solve."""
    kind = case["kind"]
    steps = 1
    if kind in ("box", "new box"):
        nod, el = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1), case["nx"] * case["ny"] * case["nz"]
        n_e, d, nip, flux, dim = 8, 3, 8, 9, 3
    elif kind == "simp":
        nod, el = (case["nx"] + 1) * (case["ny"] + 1), case["nx"] * case["ny"]
        n_e, d, nip, flux, dim = 4, 2, 4, 4, 2
    elif kind == "hyper":
        cells = case["nx"] * case["ny"] * case["nz"]
        nod, el = (2 * case["nx"] + 1) * (2 * case["ny"] + 1) * (2 * case["nz"] + 1), 6 * cells
        n_e, d, nip, flux, dim, steps = 10, 3, 4, 9, 3, 10
    elif kind == "plate":
        nod, el = case["n_theta"] * (case["n_rad"] + 1), case["n_theta"] * case["n_rad"]
        n_e, d, nip, flux, dim, steps = 4, 2, 4, 4, 2, 5
    elif kind == "roof":
        nod, el = case["n_arc"] * case["n_len"], 2 * (case["n_arc"] - 1) * (case["n_len"] - 1)
        n_e, d, nip, flux, dim = 3, 6, 3, 4, 3
    elif kind == "slab":
        nod, el = 2 * (case["n"] + 1) * (case["n"] // 2 + 1), case["n"] * (case["n"] // 2)
        n_e, d, nip, flux, dim = 8, 1, 8, 3, 3
    else:
        nod, el = (case["nx"] + 1) * (case["ny"] + 1), case["nx"] * case["ny"]
        n_e, d, nip, flux, dim, steps = 4, 1, 4, 2, 2, case["steps"]
    mesh_bytes = 8 * dim * nod + 8 * n_e * el
    field_bytes = 9 * d * nod + 8 * d * nod + 8 * el
    out_bytes = 8 * (2 * d * nod + 2 * flux * el + el)
    pairs = n_e * (n_e + 1) // 2
    element = 2 * nip * pairs * d * dim
    return {"bytes": mesh_bytes + field_bytes + out_bytes, "flops": steps * el * (element + 4 * (n_e * d) ** 2)}


# ------------------------------------------------------------------- exact --
def _shape_gradients(n_e, dim):
    """dN/dxi [nip, dim, n_e] and weights of the 2-point Gauss rules of the
    multilinear elements and of the 4-point rule of the 10-node tetrahedron
    (with the 8-digit points that the element is defined with)."""
    if n_e == 10:
        a, b = 0.58541020, 0.13819660
        pts = torch.tensor([[a, b, b], [b, a, b], [b, b, a], [b, b, b]], dtype=F64)
        w = torch.full((4,), 0.041666667, dtype=F64)

        def shape(p):
            x, y, z = p
            v = 1 - x - y - z
            return torch.stack([v * (2 * v - 1), x * (2 * x - 1), y * (2 * y - 1), z * (2 * z - 1), 4 * x * v,
                                4 * x * y, 4 * y * v, 4 * z * v, 4 * x * z, 4 * y * z])
    else:
        corner = torch.tensor([[-1, -1], [1, -1], [1, 1], [-1, 1]], dtype=F64)
        if dim == 3:
            corner = torch.cat([torch.cat([corner, torch.full((4, 1), c, dtype=F64)], 1) for c in (-1.0, 1.0)])
        g = 1.0 / math.sqrt(3.0)
        pts = torch.tensor(list(itertools.product((-g, g), repeat=dim)), dtype=F64)
        w = torch.ones(len(pts), dtype=F64)

        def shape(p):
            return (1 + corner * p).prod(1) / 2**dim
    return torch.stack([torch.autograd.functional.jacobian(shape, p).T for p in pts]).cuda(), w.cuda()


class _Plain:
    """Plain torch restatement of a linear analysis with elements that share
    one type: element matrices by einsum, matrix-free products, Jacobi CG in
    64 bits run to its rounding floor."""

    def __init__(self, nodes, el, d):
        self.el, self.d, self.n = el, d, len(nodes) * d
        dn, self.w = _shape_gradients(el.shape[1], nodes.shape[1])
        J = torch.einsum("qia,eaj->qeij", dn, nodes[el])
        self.detw = torch.linalg.det(J) * self.w[:, None]
        self.B = torch.linalg.solve(J, dn[:, None].expand(-1, len(el), -1, -1))  # [q, e, j, a]
        self.idx = (el[:, :, None] * d + torch.arange(d, device=el.device)).reshape(len(el), -1)

    def scatter(self, fe):
        return torch.zeros(self.n, dtype=F64, device=fe.device).index_add_(0, self.idx.ravel(), fe.ravel())

    def iso(self, lam, G):
        """Element matrices of lam tr(e) I + 2 G e."""
        M = torch.einsum("qe,qeia,qekb->eaibk", self.detw, self.B, self.B)
        K = lam[:, None, None, None, None] * M + G[:, None, None, None, None] * M.transpose(2, 4)
        tr = torch.einsum("eaibi->eab", M)
        K += torch.einsum("eab,ik->eaibk", G[:, None, None] * tr, torch.eye(self.d, dtype=F64, device=M.device))
        return K.reshape(len(M), self.idx.shape[1], -1)

    def conduct(self, kappa):
        return torch.einsum("qe,qeia,qeib->eab", self.detw * kappa, self.B, self.B)

    def apply(self, Ke, x):
        return self.scatter(torch.bmm(Ke, x[self.idx][:, :, None]))

    def cg(self, Ke, b, con):
        diag = self.scatter(torch.diagonal(Ke, dim1=1, dim2=2).contiguous())
        free = (~con).to(F64)
        minv = free / diag
        b = b * free
        x = torch.zeros_like(b)
        for _ in range(3):  # restarts on the true residual reach the rounding floor
            r = b - free * self.apply(Ke, x)
            stop = 1e-14 * float(b.norm())
            z = minv * r
            p, rz = z, torch.dot(r, z)
            for it in range(20000):
                q = free * self.apply(Ke, p)
                a = rz / torch.dot(p, q)
                x = x + a * p
                r = r - a * q
                if it % 25 == 24 and float(r.norm()) <= stop:
                    break
                z = minv * r
                rz, old = torch.dot(r, z), rz
                p = z + (rz / old) * p
        return x

    def gradient(self, x):
        """dx_c / dX_j at the points, [q, e, c, j]."""
        return torch.einsum("eac,qeja->qecj", x.reshape(-1, self.d)[self.el], self.B)


def _exact_linear(case, d):
    kind = case["kind"]
    nodes, el, con = d["nodes"], d["el"], d["con"].ravel()
    if kind == "slab":
        P = _Plain(nodes, el, 1)
        k = 1e-3 + (1.0 - 1e-3) * d["rho"] ** 3
        Ke = P.conduct(k)
        T = P.cg(Ke, d["q"].ravel(), con)
        h = P.gradient(T)[:, :, 0].mean(0)
        Te = T[P.idx]
        g = -torch.einsum("ea,eab,eb->e", Te, Ke, Te) / k * (1.0 - 1e-3) * 3 * d["rho"] ** 2
        return {"T": T[:, None], "f": P.apply(Ke, T)[:, None], "q": k[:, None] * h, "grad": h, "g": g}
    dim = nodes.shape[1]
    P = _Plain(nodes, el, dim)
    E, nu = (d["E"] if "E" in d else d["rho"] ** 3), float(NU)
    G = E / (2 * (1 + nu))
    lam = E * nu / ((1 + nu) * (1 - 2 * nu)) if dim == 3 else E * nu / (1 - nu**2)
    Ke = P.iso(lam, G)
    u = P.cg(Ke, d["forces"].ravel(), con)
    H = P.gradient(u).mean(0)
    eps = 0.5 * (H + H.transpose(1, 2))
    eye = torch.eye(dim, dtype=F64, device=H.device)
    s = lam[:, None, None] * torch.einsum("eii->e", eps)[:, None, None] * eye + 2 * G[:, None, None] * eps
    if case.get("wrt") == "forces":
        g = P.cg(Ke, torch.ones_like(u), con).reshape(-1, dim)
    else:
        ue = u[P.idx]
        g = -torch.einsum("ea,eab,eb->e", ue, Ke, ue) / E
        if kind == "simp":
            g = g * 3 * d["rho"] ** 2
    return {"u": u.reshape(-1, dim), "f": P.apply(Ke, u).reshape(-1, dim), "s": s, "F": H + eye, "g": g}


def _exact_hyper(d):
    """Equilibrium of the pulled box by a dense Newton iteration (the state is
    path-independent), and the reaction's gradient by a dense adjoint."""
    P = _Plain(d["nodes"], d["el"], 3)
    E, nu = d["E"], 0.45
    mu, lam = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
    right = d["nodes"][:, 0] == 3.0
    con = torch.zeros(P.n // 3, 3, dtype=torch.bool, device=mu.device)
    con[d["nodes"][:, 0] == 0.0] = True
    con[right, 0] = True
    free = (~con.ravel()).nonzero().ravel()
    eye = torch.eye(3, dtype=F64, device=mu.device)

    def state(u):
        F = P.gradient(u) + eye
        Fi, J = torch.linalg.inv(F), torch.linalg.det(F)
        lnJ = torch.log(J)[..., None, None]
        pk = mu[:, None, None] * (F - Fi.transpose(-1, -2)) + lam[:, None, None] * lnJ * Fi.transpose(-1, -2)
        fe = torch.einsum("qe,qeja,qecj->eac", P.detw, P.B, pk)
        return F, Fi, J, lnJ, pk, fe

    def tangent(Fi, lnJ):
        c = (mu[:, None, None] - lam[:, None, None] * lnJ)[..., None, None]
        A = lam[:, None, None, None, None] * torch.einsum("qeji,qelk->qeijkl", Fi, Fi)
        A = A + c * torch.einsum("qejk,qeli->qeijkl", Fi, Fi)
        A = A + mu[:, None, None, None, None] * torch.einsum("ik,jl->ijkl", eye, eye)
        Ke = torch.einsum("qe,qeja,qeijkl,qelb->eaibk", P.detw, P.B, A, P.B).reshape(len(mu), 30, 30)
        K = torch.zeros(P.n, P.n, dtype=F64, device=mu.device)
        rows = P.idx[:, :, None].expand(-1, -1, 30)
        K.index_put_((rows.ravel(), P.idx[:, None, :].expand(-1, 30, -1).ravel()), Ke.ravel(), accumulate=True)
        return K

    # start from the uniform stretch, then load steps are not needed
    x = d["nodes"]
    u = torch.zeros_like(x)
    u[:, 0] = 0.5 * x[:, 0] / 3.0
    u = u.ravel()
    for _ in range(30):
        F, Fi, J, lnJ, pk, fe = state(u)
        r = P.scatter(fe)
        K = tangent(Fi, lnJ)
        du = torch.linalg.solve(K[free][:, free], r[free])
        u = u.index_add(0, free, -du)
        if float(du.norm()) <= 1e-14 * float(u.norm()):
            break
    F, Fi, J, lnJ, pk, fe = state(u)
    K = tangent(Fi, lnJ)
    v = torch.zeros(P.n // 3, 3, dtype=F64, device=mu.device)
    v[right, 0] = 1.0
    v = v.ravel()
    v = v.index_add(0, free, -torch.linalg.solve(K[free][:, free], (K @ v)[free]))
    g = (v[P.idx] * fe.reshape(len(mu), -1)).sum(1) / E
    sig = torch.einsum("qeik,qekj->qeij", F, pk) / J[..., None, None]
    return {"u": u.reshape(-1, 3), "f": P.scatter(fe).reshape(-1, 3), "s": sig.mean(0), "F": F.mean(0), "g": g}


def exact(case, seed):
    """The outputs in 64 bits by plain torch: linear analyses and the
    hyperelastic one.  The plate (path-dependent plasticity), the shell and
    the transient have no such short restatement."""
    kind = case["kind"]
    if kind in ("box", "new box", "simp", "slab"):
        return _exact_linear(case, _inputs(case, seed))
    if kind == "hyper":
        return _exact_hyper(_inputs(case, seed))
    return None
