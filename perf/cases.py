"""Performance cases of the operator / solver library: what a simulation program calls, over real sizes.

Every case goes through meltpooldg_b200.operators (or .adjoint) on device vectors, as the time loop of a
melt-pool or level-set program does.  `listed` are fixed cases, `draw` makes more of the same ranges,
`exact` evaluates the same weak forms in plain torch in 64 bits (cell views, 1-D tables, strided adds).

Kinds:
  vmult       heat operator apply, the inner call of every Krylov iteration (FE_Q(1..4), FP64 / FP32)
  newton      what one Newton step of the heat equation evaluates besides its linear solve: residual,
              Jacobi diagonal and one tangent apply, with convection and radiation on the top face and
              a constant or a solid / liquid material
  advection   level-set advection-diffusion apply (affine or DoF-vector velocity, with or without SUPG)
  reinit      reinitialisation (Olsson): right-hand side and one tangent apply
  projection  normal-vector and curvature right-hand sides and one projection apply, optional narrow band
  cg / mixed  linear solve of an implicit heat step: FP64 Jacobi-CG / FP32 inner CG in FP64 defect correction
  gmres       one implicit level-set advection step: right-hand side and Jacobi-GMRES(30)
  adjoint     objective and gradient of a transient heat problem (forward and backward sweep)
"""
import math

import numpy as np
import torch

from meltpooldg_b200.adjoint import TransientHeatAdjoint
from meltpooldg_b200.operators import (AdvectionDiffusionOperator, HeatDiffuseOperator, LinearSolver,
                                       LinearSolverData, Mesh, OlssonOperator)


def listed():
    return [
        # the smallest call: one apply of the 16^3 FE_Q(2) heat operator (latency and launches)
        _case("heat_q2_16_f64", "vmult", 2, (16, 16, 16), dtype="f64", field=False),
        # the benchmark's headline apply: FE_Q(4), 17.0 M DoFs, per-cell conductivity
        _case("heat_q4_64_f64", "vmult", 4, (64, 64, 64), dtype="f64", field=True),
        # an ordinary FP32 apply (inner operator of the mixed solver) on a ragged, odd mesh
        _case("heat_q2_ragged_f32", "vmult", 2, (131, 97, 118), dtype="f32", field=True),
        # Newton step of a conduction problem with radiation, FE_Q(1) on a large plate
        _case("newton_q1_faces_f64", "newton", 1, (192, 160, 72), solid=False),
        # Newton step through the mushy zone (solid / liquid material with latent heat)
        _case("newton_q2_solid_f64", "newton", 2, (80, 64, 48), solid=True),
        # level-set advection apply of the benchmark's time step
        _case("advection_q2_96_f64", "advection", 2, (96, 96, 96), dtype="f64", velocity="affine", supg=False),
        # stabilised advection with the flow solver's velocity, FP32 inner operator, ragged
        _case("advection_q2_supg_f32", "advection", 2, (61, 90, 77), dtype="f32", velocity="field", supg=True),
        # one pseudo-time step of the reinitialisation
        _case("reinit_q2_f64", "reinit", 2, (72, 56, 64)),
        # normal and curvature of the interface in a narrow band
        _case("projection_q2_f64", "projection", 2, (57, 83, 71), band=True),
        # the benchmark's linear solve: FE_Q(2), 17.0 M DoFs, mixed precision
        _case("mixed_q2_128", "mixed", 2, (128, 128, 128)),
        # one implicit advection step
        _case("gmres_q2_64", "gmres", 2, (64, 64, 64), velocity="affine", supg=False),
        # gradient of a transient heat problem
        _case("adjoint_q2_32", "adjoint", 2, (32, 32, 32), steps=6),
    ]


def draw(rng):
    kind = rng.choice(["vmult"] * 4 + ["newton"] * 3 + ["advection"] * 3 + ["reinit"] * 2 + ["projection"] * 2 +
                      ["cg", "mixed", "gmres", "adjoint"])
    degree = rng.choice({"vmult": (1, 2, 2, 3, 4, 4), "cg": (1, 2, 2, 3, 4), "mixed": (1, 2, 2, 3, 4),
                         "adjoint": (1, 2)}.get(kind, (1, 1, 2, 2, 2, 3)))
    most = {"vmult": 1.7e7, "newton": 2.2e6, "advection": 7.2e6, "reinit": 2.2e6, "projection": 2.8e6, "cg": 6e6,
            "mixed": 1.0e7, "gmres": 1.5e6, "adjoint": 2.6e5}[kind]
    while True:
        side = math.exp(rng.uniform(math.log(3e4), math.log(most)) / 3) / degree
        cells = tuple(max(4, round(side * rng.uniform(0.65, 1.5))) for _ in range(3))
        if math.prod(degree * c + 1 for c in cells) <= most:
            break
    more = {"vmult": lambda: {"dtype": rng.choice(("f64", "f64", "f32")), "field": rng.random() < 0.7},
            "newton": lambda: {"solid": degree <= 3 and rng.random() < 0.6},
            "advection": lambda: {"dtype": rng.choice(("f64", "f64", "f32")),
                                  "velocity": rng.choice(("affine", "field")), "supg": rng.random() < 0.4},
            "projection": lambda: {"band": rng.random() < 0.5},
            "gmres": lambda: {"velocity": rng.choice(("affine", "field")), "supg": False},
            "adjoint": lambda: {"steps": rng.randint(3, 6)}}.get(kind, dict)()
    return _case(None, kind, degree, cells, **more)


def _case(name, kind, degree, cells, **more):
    case = {"kind": kind, "degree": degree, "mx": cells[0], "my": cells[1], "mz": cells[2], **more}
    return case if name is None else {"name": name, **case}


# ---------------------------------------------------------------------------------------------------
# physical parameters of the kinds

HEAT_DT = 1e-3                      # unit cube, rho c_p = 1 (vmult, cg, mixed, adjoint)
PLATE = 1.0e-3                      # newton: x extent in m, SI units, a titanium alloy
SOLID, LIQUID = (4400.0, 700.0, 25.0), (4100.0, 850.0, 30.0)  # density, specific heat, conductivity
T_SOLIDUS, T_LIQUIDUS, LATENT = 1800.0, 2000.0, 2.9e5
H_CONV, T_INF, EMISSIVITY, STEFAN_BOLTZMANN, DT_SI = 40.0, 300.0, 0.4, 5.670374419e-8, 1e-6
ADV_DT, ADV_EPS = 5e-3, 1e-3        # advection by a rotation about the cube's axis
ROTATION = (0.5, -0.5, 0.0, 0.0, -1.0, 0.0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0)  # v = v0 + G x, rows of G
DIRICHLET = {"newton": 16, "advection": 3, "gmres": 3, "reinit": 0, "projection": 0}  # otherwise every face
TOP = 32                            # newton: the face with convection and radiation
NORMAL_TOL = 1e-10
SOLVE_TOL = 1e-12                   # the library's default relative tolerance
MIXED_TOL, MIXED_INNER = 1e-11, 1e-5


def _box(case):
    k, m = case["degree"], (case["mx"], case["my"], case["mz"])
    size = PLATE if case["kind"] == "newton" else 1.0
    length = (size, size * m[1] / m[0], size * m[2] / m[0]) if case["kind"] == "newton" else (1.0, 1.0, 1.0)
    return Mesh(k, m, length=length, dirichlet_faces=DIRICHLET.get(case["kind"], 63))


def _spacing(mesh):
    return [length / m for length, m in zip(mesh.length, mesh.cells)]


def _coordinates(mesh):
    """x, y, z of the support points, broadcastable against [nz, ny, nx]."""
    nodes, out = _tables(mesh.degree)["nodes"], []
    for h, m in zip(_spacing(mesh), mesh.cells):
        x = (torch.arange(m, dtype=torch.float64, device="cuda")[:, None] + nodes[None, :-1]).reshape(-1)
        out.append(h * torch.cat([x, torch.tensor([float(m)], dtype=torch.float64, device="cuda")]))
    x, y, z = out
    return x[None, None, :], y[None, :, None], z[:, None, None]


def _inputs(case, seed):
    """The device tensors that a program holds before the call, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    mesh, kind = _box(case), case["kind"]
    shape, cells = mesh.n[::-1], mesh.cells[::-1]
    uniform = lambda lo, hi: lo + (hi - lo) * torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)  # noqa: E731
    number = lambda lo, hi: lo + (hi - lo) * float(torch.rand((), generator=gen, device="cuda", dtype=torch.float64))  # noqa: E731
    d = {}
    if kind in ("vmult", "cg", "mixed"):
        d["src"] = uniform(-1.0, 1.0).to(torch.float32 if case.get("dtype") == "f32" else torch.float64)
        if kind != "vmult":  # a right-hand side is 0 on the constrained rows (every face)
            d["src"] = torch.nn.functional.pad(d["src"][1:-1, 1:-1, 1:-1], (1,) * 6)
        if case.get("field", True):
            d["k"] = torch.exp(0.5 * torch.randn(cells, generator=gen, device="cuda", dtype=torch.float64))
    elif kind == "newton":
        x, y, z = _coordinates(mesh)
        lx, ly, lz = mesh.length
        cx, cy, wide = number(0.3, 0.7) * lx, number(0.3, 0.7) * ly, number(0.15, 0.3) * lx
        spot = torch.exp(-2.0 * ((x - cx) ** 2 + (y - cy) ** 2 + (z - lz) ** 2) / wide ** 2)
        d["T_old"] = 300.0 + 2500.0 * spot + uniform(-5.0, 5.0)
        d["T"] = d["T_old"] + 60.0 * spot + uniform(-5.0, 5.0)
        d["q"] = 1e14 * spot  # heat source in W/m^3
        d["src"] = uniform(-1.0, 1.0)
    elif kind == "adjoint":
        x, y, z = _coordinates(mesh)
        d["z"] = 0.3 * torch.randn(cells, generator=gen, device="cuda", dtype=torch.float64)
        y0 = number(0.4, 0.6)
        d["qhat"] = torch.stack([torch.exp(-2.0 * ((x - 0.2 - 0.05 * s) ** 2 + (y - y0) ** 2 + (z - 0.9) ** 2) / 0.2 ** 2)
                                 for s in range(case["steps"])])
        d["target"] = torch.stack([0.05 * uniform(0.0, 1.0) for _ in range(case["steps"])])
    else:  # level-set kinds: a smeared sphere, the velocity or the normal field
        x, y, z = _coordinates(mesh)
        cx, cy, cz, radius = number(0.4, 0.6), number(0.6, 0.75), number(0.4, 0.6), number(0.15, 0.25)
        dist = torch.sqrt((x - cx) ** 2 + (y - cy) ** 2 + (z - cz) ** 2)
        eps = 1.5 * max(_spacing(mesh))
        d["phi"] = torch.tanh((radius - dist) / eps)
        if kind == "gmres":
            d["phi"] = d["phi"] + uniform(-1e-3, 1e-3)
        if case.get("velocity") == "field":
            w = number(0.8, 1.2)
            d["v"] = [w * (0.5 - y) + 0.1 * torch.sin(6.0 * z) + uniform(-0.01, 0.01),
                      w * (x - 0.5) + 0.1 * torch.cos(5.0 * x) + uniform(-0.01, 0.01), 0.2 * torch.sin(4.0 * y) + uniform(-0.01, 0.01)]
        if kind in ("reinit", "projection"):
            d["n"] = [(c - p) / (dist + 0.05) + uniform(-0.02, 0.02) for c, p in ((cx, x), (cy, y), (cz, z))]
        if kind != "gmres":
            d["src"] = (d["phi"] + uniform(-0.1, 0.1)).to(torch.float32 if case.get("dtype") == "f32" else torch.float64)
    flat = lambda v: [flat(t) for t in v] if isinstance(v, list) else v.contiguous().reshape(-1)  # noqa: E731
    return mesh, {key: flat(v) for key, v in d.items()}


def prepare(case, seed):
    mesh, d = _inputs(case, seed)
    kind = case["kind"]
    empty = lambda: torch.empty(mesh.ndofs, dtype=torch.float64, device="cuda")  # noqa: E731
    s = {"case": case, "in": d}
    if kind in ("vmult", "cg", "mixed", "adjoint"):
        op = HeatDiffuseOperator(mesh, rho_cp=1.0, dt=HEAT_DT, conductivity=1.0)
        if "k" in d:
            op.set_conductivity(d["k"])
        if kind == "vmult":
            s["dst"] = torch.empty_like(d["src"])
        elif kind == "adjoint":
            s["adjoint"] = TransientHeatAdjoint(op, n_steps=case["steps"], checkpoint_every=3)
            s["grad"] = torch.empty(mesh.ncells, dtype=torch.float64, device="cuda")
        else:
            s["x"] = empty()
    elif kind == "newton":
        op = HeatDiffuseOperator(mesh, rho_cp=SOLID[0] * SOLID[1], dt=DT_SI, conductivity=SOLID[2])
        op.set_boundary_conditions(convection_faces=TOP, convection_coefficient=H_CONV,
                                   convection_temperature_infinity=T_INF, radiation_faces=TOP, emissivity=EMISSIVITY,
                                   radiation_temperature_infinity=T_INF)
        if case["solid"]:
            op.set_solidification(liquid=LIQUID, solid=SOLID, liquidus_temperature=T_LIQUIDUS,
                                  solidus_temperature=T_SOLIDUS, latent_heat=LATENT)
        op.set_temperature(d["T"])
        op.set_old_temperature(d["T_old"])
        s["rhs"], s["diag"], s["dst"] = empty(), empty(), empty()
    elif kind in ("advection", "gmres"):
        op = AdvectionDiffusionOperator(mesh, dt=ADV_DT, theta=1.0, diffusivity=ADV_EPS, velocity=ROTATION)
        if "v" in d:
            op.set_velocity_field(*d["v"])
        if case["supg"]:
            op.set_convection_stabilization("SUPG", -1.0)
        if kind == "advection":
            s["dst"] = torch.empty_like(d["src"])
        else:
            s["rhs"], s["x"] = empty(), empty()
    elif kind == "reinit":
        h = max(_spacing(mesh))
        op = OlssonOperator(mesh, dt=0.5 * h, eps_normal=h, eps_tangential=0.25 * h, normal_tolerance=NORMAL_TOL)
        op.set_normal(*d["n"])
        s["rhs"], s["dst"] = empty(), empty()
    else:  # projection: M + damping K
        op = HeatDiffuseOperator(mesh, rho_cp=1.0, dt=1.0, conductivity=max(_spacing(mesh)) ** 2)
        if case["band"]:
            op.set_narrow_band(d["phi"], _band())
        s["normal"], s["curvature"], s["dst"] = [empty() for _ in range(3)], empty(), empty()
    s["op"] = op
    return s


def _band():
    return 0.95  # |level set| below which a point belongs to the narrow band


def run(state):
    case, op, d = state["case"], state["op"], state["in"]
    kind = case["kind"]
    if kind in ("vmult", "advection"):
        op.vmult(state["dst"], d["src"])
        return state["dst"]
    if kind == "newton":
        state["rhs"].zero_()
        op.create_rhs(state["rhs"], d["T"], d["T_old"], d["q"])
        op.compute_inverse_diagonal_from_matrixfree(state["diag"])
        op.vmult(state["dst"], d["src"])
        return {"rhs": state["rhs"], "diag": state["diag"], "dst": state["dst"]}
    if kind == "reinit":
        op.create_rhs(state["rhs"], d["phi"])
        op.vmult(state["dst"], d["src"])
        return {"rhs": state["rhs"], "dst": state["dst"]}
    if kind == "projection":
        for n in state["normal"]:
            n.zero_()
        op.level_set_normal_rhs(d["phi"], *state["normal"])
        op.level_set_curvature_rhs(state["curvature"], *d["n"], NORMAL_TOL)
        op.vmult(state["dst"], d["src"])
        return {"normal": state["normal"], "curvature": state["curvature"], "dst": state["dst"]}
    if kind == "cg":
        state["x"].zero_()
        LinearSolver.solve(op, state["x"], d["src"], LinearSolverData("CG", "Diagonal", rel_tolerance=SOLVE_TOL))
        return state["x"]
    if kind == "mixed":
        state["x"].zero_()
        LinearSolver.solve_mixed(op, state["x"], d["src"], outer_rel_tol=MIXED_TOL, inner_rel_tol=MIXED_INNER)
        return state["x"]
    if kind == "gmres":
        state["rhs"].zero_()
        op.create_rhs(state["rhs"], d["phi"])
        state["x"].copy_(d["phi"])
        LinearSolver.solve(op, state["x"], state["rhs"], LinearSolverData("GMRES", "Diagonal", rel_tolerance=SOLVE_TOL))
        return {"rhs": state["rhs"], "x": state["x"]}
    J, dA, _ = state["adjoint"].objective_and_gradient(d["z"], d["qhat"], 10.0, d["target"], state["grad"])
    return {"J": J, "dA": dA, "grad": state["grad"]}


def work(case):
    """Inputs read once and outputs written once per operator call; sum factorisation's operations.

    A solve counts its iterations' vectors (5 read, 4 written) at the usual number of iterations."""
    mesh, kind, n = _box(case), case["kind"], case["degree"] + 1
    N, C, word = mesh.ndofs, mesh.ncells, 4 if case.get("dtype") == "f32" else 8
    sweep = 2 * n ** 4 * C  # one 1-D transform of every cell
    apply = 6 * sweep + 2 * n ** 3 * C
    if kind == "vmult":
        return {"bytes": word * (2 * N + (C if case["field"] else 0)), "flops": apply}
    if kind == "newton":
        fields = 3 if case["solid"] else 1  # T and T_old are read by the tangent and its diagonal, too
        return {"bytes": 8 * N * (4 + fields + 1 + fields), "flops": 3 * apply}
    if kind == "advection":
        return {"bytes": N * (2 * word + (24 if case["velocity"] == "field" else 0)), "flops": 2 * apply}
    if kind == "reinit":
        return {"bytes": 8 * N * 10, "flops": 4 * apply}
    if kind == "projection":
        return {"bytes": 8 * N * (10 if case["band"] else 8), "flops": 4 * apply}
    if kind == "adjoint":
        solves, iterations = 3 * case["steps"], 25
        return {"bytes": 8 * (9 * N + C) * solves * iterations, "flops": apply * solves * iterations}
    iterations = {"cg": 60, "mixed": 250, "gmres": 25}[kind]
    per = {"cg": 8 * (9 * N + C), "mixed": 4 * (9 * N + C), "gmres": 8 * (2 * N + iterations * N)}[kind]
    return {"bytes": per * iterations, "flops": (apply + 2 * 14 * N) * iterations}


# ---------------------------------------------------------------------------------------------------
# the same forms in plain torch, 64 bits

_TABLES = {}


def _tables(k):
    """FE_Q(k) on [0, 1]: Gauss-Lobatto nodes; values, first and second derivatives at the k + 1 Gauss points."""
    if k not in _TABLES:
        inner = np.polynomial.legendre.Legendre.basis(k).deriv().roots() if k > 1 else np.zeros(0)
        nodes = 0.5 * (1.0 + np.concatenate([[-1.0], np.sort(inner.real), [1.0]]))
        q, w = np.polynomial.legendre.leggauss(k + 1)
        q, w = 0.5 * (1.0 + q), 0.5 * w
        coefficients = np.linalg.inv(np.vander(nodes, increasing=True))  # columns: the Lagrange polynomials
        power = np.vander(q, k + 1, increasing=True)
        first, second = np.zeros_like(power), np.zeros_like(power)
        for p in range(1, k + 1):
            first[:, p] = p * q ** (p - 1)
        for p in range(2, k + 1):
            second[:, p] = p * (p - 1) * q ** (p - 2)
        arrays = {"nodes": nodes, "q": q, "w": w, "B": power @ coefficients, "G": first @ coefficients,
                  "H": second @ coefficients}
        _TABLES[k] = {key: torch.tensor(v, device="cuda", dtype=torch.float64) for key, v in arrays.items()}
    return _TABLES[k]


class _Forms:
    """Cell integrals of one mesh; cell arrays are [mz, my, mx, z, y, x]."""

    def __init__(self, mesh):
        self.mesh, self.k, self.n = mesh, mesh.degree, mesh.degree + 1
        self.h, self.t = _spacing(mesh), _tables(mesh.degree)
        w = self.t["w"]
        self.jxw = math.prod(self.h) * w[:, None, None] * w[None, :, None] * w[None, None, :]
        self.free = torch.ones(mesh.n[::-1], dtype=torch.bool, device="cuda")
        for f in range(6):
            if mesh.dirichlet_faces >> f & 1:
                self.free.select(2 - f // 2, -1 if f % 2 else 0).fill_(False)

    def masked(self, u):
        return torch.where(self.free, u.double().view(self.free.shape), 0.0)

    def cells(self, u):
        u = u.double().view(self.free.shape)
        for dim in range(3):
            u = u.unfold(dim, self.n, self.k)
        return u

    @staticmethod
    def along(u, mz, my, mx):
        u = torch.matmul(u, mx.T)
        u = torch.matmul(my, u)
        return torch.einsum("...zyx,az->...ayx", u, mz)

    def value(self, u):
        B = self.t["B"]
        return self.along(self.cells(u), B, B, B)

    def gradient(self, u):
        B, G, u = self.t["B"], self.t["G"], self.cells(u)
        return [self.along(u, *([G if e == d else B for e in (2, 1, 0)])) / self.h[d] for d in range(3)]

    def laplacian(self, u):
        B, H, u = self.t["B"], self.t["H"], self.cells(u)
        return sum(self.along(u, *([H if e == d else B for e in (2, 1, 0)])) / self.h[d] ** 2 for d in range(3))

    def assemble(self, cell):
        out = torch.zeros(self.free.shape, dtype=torch.float64, device="cuda")
        m = self.mesh.cells[::-1]
        at = lambda i, dim: slice(i, i + self.k * (m[dim] - 1) + 1, self.k)  # noqa: E731
        for a in range(self.n):
            for b in range(self.n):
                for c in range(self.n):
                    out[at(a, 0), at(b, 1), at(c, 2)] += cell[..., a, b, c]
        return out

    def test(self, value=None, flux=None):
        """int value phi + flux . grad phi on the free rows."""
        B, G, cell = self.t["B"].T, self.t["G"].T, 0.0
        if value is not None:
            cell = cell + self.along(value * self.jxw, B, B, B)
        if flux is not None:
            for d in range(3):
                cell = cell + self.along(flux[d] * self.jxw, *([G if e == d else B for e in (2, 1, 0)])) / self.h[d]
        return torch.where(self.free, self.assemble(cell), 0.0)

    def diagonal(self, mass, stiffness, mixed):
        """int mass phi_i^2 + stiffness |grad phi_i|^2 + (mixed . grad phi_i) phi_i for every basis function."""
        B, G = self.t["B"].T, self.t["G"].T
        BB, GG, BG = B * B, G * G, B * G
        cell = self.along(mass * self.jxw, BB, BB, BB)
        for d in range(3):
            cell = cell + self.along(stiffness * self.jxw, *([GG if e == d else BB for e in (2, 1, 0)])) / self.h[d] ** 2
            if mixed is not None:
                cell = cell + self.along(mixed[d] * self.jxw, *([BG if e == d else BB for e in (2, 1, 0)])) / self.h[d]
        return self.assemble(cell)

    # the top face (z high): values at its Gauss points, and their test
    def top(self, u):
        u = u.double().view(self.free.shape)[-1].unfold(0, self.n, self.k).unfold(1, self.n, self.k)
        return torch.matmul(self.t["B"], torch.matmul(u, self.t["B"].T))

    def test_top(self, value, table):
        w = self.t["w"][:, None] * self.t["w"][None, :] * self.h[0] * self.h[1]
        cell = torch.matmul(table.T, torch.matmul(value * w, table))
        out = torch.zeros_like(self.free, dtype=torch.float64)
        m = self.mesh.cells
        for b in range(self.n):
            for c in range(self.n):
                out[-1, b:b + self.k * (m[1] - 1) + 1:self.k, c:c + self.k * (m[0] - 1) + 1:self.k] += cell[..., b, c]
        return torch.where(self.free, out, 0.0)


class _Heat(_Forms):
    """rho c_p / dt M + K(k) with a conductivity per cell, by the dense cell matrices of the box."""

    def __init__(self, mesh, k=None):
        super().__init__(mesh)
        B, G, w = self.t["B"], self.t["G"], self.t["w"]
        M, K = B.T @ (w[:, None] * B), G.T @ (w[:, None] * G)
        three = lambda a, b, c: torch.kron(torch.kron(a, b), c)  # noqa: E731
        hx, hy, hz = self.h
        self.M = hx * hy * hz * three(M, M, M)
        self.K = hy * hz / hx * three(M, M, K) + hx * hz / hy * three(M, K, M) + hx * hy / hz * three(K, M, M)
        self.kc = (torch.ones(mesh.ncells, dtype=torch.float64, device="cuda") if k is None else k).view(-1, 1)

    def _rows(self, cell):
        n = self.n
        return torch.where(self.free, self.assemble(cell.view(*self.mesh.cells[::-1], n, n, n)), 0.0)

    def _flat(self, u):
        return self.cells(u).reshape(-1, self.n ** 3)

    def apply(self, u, rho_cp_dt=1.0 / HEAT_DT):
        u = self._flat(self.masked(u))
        return self._rows(torch.addmm((u @ self.K).mul_(self.kc), u, self.M, alpha=rho_cp_dt))

    def mass(self, u):
        return self._rows(self._flat(u) @ self.M)

    def stiffness_form(self, a, b):
        return ((self._flat(a) @ self.K) * self._flat(b)).sum(1)

    def solve(self, b, rounds=2000):
        """CG with the cells' diagonal to rounding."""
        diag = self._rows((self.kc * self.K.diagonal() + self.M.diagonal() / HEAT_DT).contiguous())
        inv = torch.where(self.free, 1.0 / diag.clamp_min(1e-300), 0.0)
        b = torch.where(self.free, b.double().view(self.free.shape), 0.0)
        x, r, p, rho, start = torch.zeros_like(b), b.clone(), 0.0, None, float(b.norm())
        for _ in range(rounds):
            if float(r.norm()) <= 1e-14 * start:
                break
            z = inv * r
            new = (r * z).sum()
            p = z if rho is None else z + (new / rho) * p
            v = self.apply(p)
            a = new / (p * v).sum()
            x, r, rho = x + a * p, r - a * v, new
        return x


def _material(T, solid):
    """rho c_p, k and their derivatives at T (cubic blend over the mushy zone, apparent capacity of the latent heat)."""
    if not solid:
        one = torch.ones_like(T)
        return SOLID[0] * SOLID[1] * one, SOLID[2] * one, 0.0 * one, 0.0 * one
    wide = T_LIQUIDUS - T_SOLIDUS
    fs = ((T_LIQUIDUS - T) / wide).clamp(0.0, 1.0)
    weight, slope = (3.0 - 2.0 * fs) * fs * fs, -(6.0 * fs - 6.0 * fs * fs) / wide
    (rho, drho), (cp, dcp), (k, dk) = [(li + (so - li) * weight, (so - li) * slope) for li, so in zip(LIQUID, SOLID)]
    # tent of height 2 L / dT, its flanks flat over dT / 6 at both ends
    half, delta, peak = 0.5 * wide, wide / 6.0, 2.0 * LATENT / wide
    x = half - (T - 0.5 * (T_SOLIDUS + T_LIQUIDUS)).abs()  # distance from the zone's nearer end
    s = peak / (half - delta)
    c = torch.where(x < delta, 0.5 * s * x * x / delta,
                    torch.where(x > half - delta, peak - 0.5 * s * (half - x) ** 2 / delta, s * (x - 0.5 * delta)))
    dc = torch.where(x < delta, s * x / delta, torch.where(x > half - delta, s * (half - x) / delta, s * torch.ones_like(x)))
    inside = x > 0.0
    c = torch.where(inside, c, 0.0)
    dc = torch.where(inside, dc * torch.sign(0.5 * (T_SOLIDUS + T_LIQUIDUS) - T), 0.0)
    cp, dcp = cp + c, dcp + dc
    return rho * cp, k, drho * cp + rho * dcp, dk


def _velocity(f, d):
    if "v" in d:
        return [f.value(v) for v in d["v"]]
    q, at = f.t["q"], []
    for e in range(3):
        x = f.h[e] * (torch.arange(f.mesh.cells[e], dtype=torch.float64, device="cuda")[:, None] + q[None, :])
        shape = [1] * 6
        shape[2 - e], shape[5 - e] = x.shape
        at.append(x.reshape(shape))
    one = torch.ones([*f.mesh.cells[::-1], f.n, f.n, f.n], dtype=torch.float64, device="cuda")
    return [one * (ROTATION[c] + sum(ROTATION[3 + 3 * c + e] * at[e] for e in range(3))) for c in range(3)]


def _advection(f, d, supg):
    v = _velocity(f, d)
    tau = 0.0
    if supg:
        speed = torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2).amax(dim=(3, 4, 5), keepdim=True)
        tau = math.sqrt(sum(h * h for h in f.h) / 3.0) / speed

    def apply(u):
        u = f.masked(u)
        value, grad = f.value(u), f.gradient(u)
        along = v[0] * grad[0] + v[1] * grad[1] + v[2] * grad[2]
        flux = [ADV_EPS * g for g in grad]
        if supg:
            residual = tau * (value / ADV_DT + along - ADV_EPS * f.laplacian(u))
            flux = [a + residual * b for a, b in zip(flux, v)]
        return f.test(value / ADV_DT + along, flux)
    return apply


def _gmres(apply, b, x, restart=60):
    start = None
    for _ in range(8):
        r = (b - apply(x)).reshape(-1)
        beta = float(r.norm())
        start = start or beta
        if beta <= 1e-14 * start:
            break
        V, H = [r / beta], np.zeros((restart + 1, restart))
        for j in range(restart):
            w = apply(V[j].view(x.shape)).reshape(-1)
            for i, vi in enumerate(V):
                H[i, j] = float(w @ vi)
                w = w - H[i, j] * vi
            H[j + 1, j] = float(w.norm())
            V.append(w / H[j + 1, j])
            e = np.zeros(j + 2)
            e[0] = beta
            y, left = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)[:2]
            if np.linalg.norm(H[:j + 2, :j + 1] @ y - e) <= 1e-15 * start:
                break
        x = x + sum(float(c) * vi for c, vi in zip(y, V)).view(x.shape)
    return x


def _unit(v):
    norm = torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
    return [c / torch.where(norm > NORMAL_TOL, norm, NORMAL_TOL) for c in v]


def exact(case, seed):
    mesh, d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "vmult":
        return _Heat(mesh, d.get("k")).apply(d["src"]).reshape(-1)
    if kind in ("cg", "mixed"):
        return _Heat(mesh, d["k"]).solve(d["src"]).reshape(-1)
    if kind == "adjoint":
        return _exact_adjoint(case, mesh, d)
    f = _Forms(mesh)
    if kind == "newton":
        return _exact_newton(case, f, d)
    if kind == "advection":
        return _advection(f, d, case["supg"])(d["src"]).reshape(-1)
    if kind == "gmres":
        rhs = f.test(f.value(d["phi"]) / ADV_DT)  # theta = 1
        # the Dirichlet values of the initial guess stay in x; the operator reads them as 0
        x = f.masked(d["phi"])
        x = torch.where(f.free, _gmres(_advection(f, d, False), rhs, x), d["phi"].view(x.shape))
        return {"rhs": rhs.reshape(-1), "x": x.reshape(-1)}
    if kind == "reinit":
        h = max(f.h)
        n = _unit([f.value(c) for c in d["n"]])

        def flux(u):
            g = f.gradient(u)
            gn = sum(a * b for a, b in zip(g, n))
            return [0.25 * h * a + 0.75 * h * gn * b for a, b in zip(g, n)]
        phi = f.value(d["phi"])
        rhs = f.test(None, [0.5 * (1.0 - phi * phi) * b - a for a, b in zip(flux(d["phi"]), n)])
        dst = f.test(f.value(d["src"]) / (0.5 * h), flux(d["src"]))
        return {"rhs": rhs.reshape(-1), "dst": dst.reshape(-1)}
    phi = f.value(d["phi"])
    band = (phi.abs() < _band()).double() if case["band"] else torch.ones_like(phi)
    normal = [f.test(g * band) for g in f.gradient(d["phi"])]
    unit = _unit(d["n"])
    divergence = sum(f.gradient(unit[e])[e] for e in range(3))
    damping = max(f.h) ** 2
    dst = f.test(f.value(d["src"]) * band, [damping * band * g for g in f.gradient(d["src"])])
    return {"normal": [n.reshape(-1) for n in normal], "curvature": -f.test(divergence * band).reshape(-1),
            "dst": dst.reshape(-1)}


def _exact_newton(case, f, d):
    T, T_old = f.value(d["T"]), f.value(d["T_old"])
    gT = f.gradient(d["T"])
    rc, k, drc, dk = _material(T, case["solid"])
    B, top = f.t["B"], f.top(d["T"])
    sigma = EMISSIVITY * STEFAN_BOLTZMANN
    face = H_CONV + 4.0 * sigma * top ** 3
    rhs = f.test(f.value(d["q"]) - rc * (T - T_old) / DT_SI, [-k * g for g in gT])
    rhs = rhs - f.test_top(sigma * (top ** 4 - T_INF ** 4) + H_CONV * (top - T_INF), B)
    capacity = (rc + drc * (T - T_old)) / DT_SI
    diag = f.diagonal(capacity, k, [dk * g for g in gT] if case["solid"] else None) + f.test_top(face, B * B)
    diag = torch.where(f.free, 1.0 / diag, 1.0)
    src = f.masked(d["src"])
    u, gu = f.value(src), f.gradient(src)
    dst = f.test(capacity * u, [k * a + dk * b * u for a, b in zip(gu, gT)])
    dst = dst + f.test_top(face * f.top(src), B)
    return {"rhs": rhs.reshape(-1), "diag": diag.reshape(-1), "dst": dst.reshape(-1)}


def _exact_adjoint(case, mesh, d):
    k = torch.exp(d["z"])
    f, steps = _Heat(mesh, k), case["steps"]
    qhat, target = d["qhat"].view(steps, *f.free.shape), d["target"].view(steps, *f.free.shape)
    T, J = [torch.zeros_like(qhat[0])], 0.0
    for s in range(steps):
        T.append(f.solve(f.mass(T[-1] / HEAT_DT + 10.0 * qhat[s])))
        J += 0.5 * float((f.masked(T[-1] - target[s]) ** 2).sum())
    lam, grad, dA = torch.zeros_like(qhat[0]), torch.zeros_like(k), 0.0
    for s in range(steps, 0, -1):
        lam = f.solve(f.mass(lam) / HEAT_DT + f.masked(T[s] - target[s - 1]))
        grad -= k * f.stiffness_form(lam, T[s])
        dA += float((lam * f.mass(qhat[s - 1])).sum())
    return {"J": J, "dA": dA, "grad": grad}
