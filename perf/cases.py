"""What the library is timed on: calls a user of the package makes, over the sizes, degrees and options it is used with.

A case is one pass through a public entry point. Most are a chunk of the device step loop as ``solve_lwfr`` runs it (the
state in, a number of CFL steps, the time back), with the state in device memory before and after, as an ensemble or a
coupled program keeps it; the others are the drop-in rhs on host arrays, the batched stepping and the gradient through
``lw_solve``. ``draw`` gives further cases of the same ranges: meshes of 8 x 8 to 512 x 512 elements, curvilinear ones of
any size, degrees 3 to 5 (the degrees of the package's configurations), both surface fluxes and speed estimates.

``exact`` restates the schemes in plain torch (float64): the Lax-Wendroff and the two-stage step on conforming and
once-refined TreeMeshes, with shock capturing and Dirichlet boundaries, and on curvilinear meshes, and the gradient by
automatic differentiation of that restatement. The MUSCL-blended and the Navier-Stokes cases have none.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "trixilw.jl_b200"))

import trixilw as tl  # noqa: E402
from trixilw import _lib  # noqa: E402

GAMMA = 1.4
# Fourier CFL limits of the scheme for N = 3, 4 and a value below them for N = 5
CFL_LIMIT = {3: 0.170, 4: 0.103, 5: 0.07}
SHOCK_CFL = 0.15


def listed():
    return [
        # the drop-in call of a host program: one rhs on host arrays, on the smallest mesh of the configurations
        {"name": "rhs_host_16_N4", "kind": "rhs", "level": 4, "N": 4, "flux": "rusanov", "speed": "naive"},
        # solve_lwfr's chunk of 64 steps on that mesh: what a step costs where launches and latency count
        {"name": "lw_16_N4", "kind": "lw", "level": 4, "N": 4, "flux": "rusanov", "speed": "naive", "steps": 64},
        # an ordinary run at degree 3 with the other flux and speed estimate
        {"name": "lw_128_N3_hll", "kind": "lw", "level": 7, "N": 3, "flux": "hll", "speed": "davis", "steps": 32},
        # the benchmark's mesh and degree: the largest state
        {"name": "lw_512_N4", "kind": "lw", "level": 9, "N": 4, "flux": "rusanov", "speed": "naive", "steps": 8},
        # a mesh as an AMR step leaves it (a refined patch and its mortars)
        {"name": "lw_amr_64_N4", "kind": "amr", "level": 6, "N": 4, "flux": "rusanov", "speed": "naive", "steps": 16},
        # the two-stage scheme
        {"name": "mdrk_256_N4", "kind": "mdrk", "level": 8, "N": 4, "flux": "rusanov", "speed": "naive", "steps": 8},
        # shocks: blended subcells between Dirichlet boundaries
        {"name": "riemann_256_N4", "kind": "riemann", "level": 8, "N": 4, "speed": "naive", "steps": 8},
        # a curvilinear StructuredMesh with odd sides
        {"name": "warped_201x167_N4", "kind": "warped", "nx": 201, "ny": 167, "N": 4, "speed": "naive", "steps": 8},
        # shocks on a curvilinear mesh, MUSCL subcells
        {"name": "blast_warped_150x133_N4", "kind": "blast", "nx": 150, "ny": 133, "N": 4, "speed": "naive", "steps": 8},
        # Navier-Stokes: the lid-driven cavity on a warped mesh, slip walls and no-slip walls
        {"name": "cavity_64_N4", "kind": "cavity", "nx": 64, "ny": 64, "N": 4, "speed": "naive", "steps": 16},
        # uneven instances of degrees 3, 4 and 5 advanced together
        {"name": "batch_64", "kind": "batch", "count": 64, "steps": 50},
        # the gradient of a misfit of the final density with respect to the initial state
        {"name": "gradient_64_N4", "kind": "gradient", "level": 6, "N": 4, "steps": 40, "every": 10},
    ]


def draw(rng):
    kind = rng.choice(["rhs", "lw", "lw", "amr", "mdrk", "riemann", "warped", "blast", "cavity", "batch", "gradient"])
    N = rng.choice([3, 4, 5])
    case = {"kind": kind, "N": N, "speed": rng.choice(["naive", "davis"])}

    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def steps(nodes, most):
        # no more nodes times steps than the largest listed case, and no more steps than a chunk
        return max(1, min(rng.randint(4, 64), most // nodes))

    n2 = (N + 1) ** 2
    if kind in ("rhs", "lw", "mdrk", "amr", "riemann"):
        case["level"] = rng.randint(3, {"rhs": 7, "lw": 9, "mdrk": 8, "amr": 7, "riemann": 8}[kind])
        if kind == "lw" and N == 5:
            case["level"] = min(case["level"], 8)
        if kind != "riemann":
            case["flux"] = rng.choice(["rusanov", "hll"])
        if kind != "rhs":
            case["steps"] = steps(4 ** case["level"] * n2, 8 * 512 * 512 * 25 // (1 if kind == "lw" else 2))
    elif kind in ("warped", "blast", "cavity"):
        case["nx"], case["ny"] = side(8, 96 if kind == "cavity" else 256), side(8, 96 if kind == "cavity" else 256)
        case["steps"] = steps(case["nx"] * case["ny"] * n2, 4 * 512 * 512 * 25)
    elif kind == "batch":
        case = {"kind": kind, "count": side(2, 64), "steps": rng.randint(10, 60)}
    else:
        case["level"] = rng.randint(4, 6)
        case["steps"] = rng.randint(8, 40)
        case["every"] = rng.randint(3, case["steps"])
    return case


# ---- inputs: meshes, initial states and boundary data, from the seed alone ---------------------------------------
def _cfl(N):
    return 0.98 * (N + 1) * CFL_LIMIT[N]


def _warp(xi, eta):
    X, Y = 10.0 * xi, 10.0 * eta
    s = np.sin(np.pi * (X + 10.0) / 10.0) * np.sin(np.pi * (Y + 10.0) / 10.0)
    return X + s, Y + s


def _cavity_map(xi, eta):
    X, Y = 0.5 * (xi + 1.0), 0.5 * (eta + 1.0)
    s = 0.05 * np.sin(np.pi * X) * np.sin(np.pi * Y)
    return X + s, Y + s


def _vortex(rng):
    return tl.IsentropicVortex(float(rng.uniform(4.0, 5.5)), center=tuple(float(c) for c in rng.uniform(-2.0, 2.0, 2)))


class _Quadrants(tl.FourQuadrantRiemann):
    """The four-quadrant problem with each state's density and pressure off by a few per cent."""

    def __init__(self, rng):
        self.states = {q: (r * rng.uniform(0.97, 1.03), a, b, p * rng.uniform(0.97, 1.03))
                       for q, (r, a, b, p) in tl.FourQuadrantRiemann.states.items()}


class _Blasts:
    """Discs of dense gas at high pressure in a thin one at rest."""

    def __init__(self, rng):
        self.discs = [(rng.uniform(-8, 8), rng.uniform(-8, 8), rng.uniform(0.8, 2.0)) for _ in range(6)]

    def __call__(self, x, y, t, eq):
        inside = np.zeros(x.shape, dtype=bool)
        for a, b, r in self.discs:
            inside |= (x - a) ** 2 + (y - b) ** 2 < r * r
        z = np.zeros(x.shape)
        return eq.prim2cons(np.where(inside, 1.0, 0.125), z, z, np.where(inside, 10.0, 1.0))


class _Eddies:
    """A few eddies in the walled cavity, Mach 0.1 or less."""

    def __init__(self, rng):
        self.a = rng.uniform(-0.3, 0.3, (3, 3))

    def __call__(self, x, y, t, eq):
        v1, v2 = np.zeros(x.shape), np.zeros(x.shape)
        for k in range(3):
            for m in range(3):
                a, p, q = self.a[k, m], np.pi * (k + 1), np.pi * (m + 1)
                v1 += a * q * np.sin(p * x) ** 2 * np.sin(q * y) * np.cos(q * y) / 10.0
                v2 -= a * p * np.sin(q * y) ** 2 * np.sin(p * x) * np.cos(p * x) / 10.0
        return eq.prim2cons(np.ones(x.shape), v1, v2, np.full(x.shape, 1.0 / (0.1 ** 2 * GAMMA)))


def _state(ic, xy, eq):
    return np.ascontiguousarray(np.transpose(ic(xy[0], xy[1], 0.0, eq), (2, 1, 0, 3))).reshape(-1)


def _mesh(case):
    kind = case["kind"]
    box = (-10.0, -10.0), (10.0, 10.0)
    if kind == "riemann":
        return tl.TreeMesh((0.0, 0.0), (1.0, 1.0), case["level"], periodicity=False)
    if kind == "amr":
        return tl.RefinedTreeMesh(*box, case["level"], ((-4.0, -4.0), (4.0, 4.0)))
    if kind in ("warped", "blast"):
        return tl.StructuredMesh((case["nx"], case["ny"]), _warp)
    if kind == "cavity":
        return tl.StructuredMesh((case["nx"], case["ny"]), _cavity_map, periodicity=False)
    return tl.TreeMesh(*box, case["level"])


def _initial(case, seed):
    rng = np.random.default_rng(seed)
    return {"riemann": _Quadrants, "blast": _Blasts, "cavity": _Eddies}.get(case["kind"], _vortex)(rng)


def _instances(case, seed):
    """The batch: sides of 8 to 64 elements, degrees 3 to 5, each its own vortex."""
    shape, rng = np.random.default_rng(case["count"]), np.random.default_rng(seed)
    eq = tl.CompressibleEulerEquations2D(GAMMA)
    out = []
    for _ in range(case["count"]):
        level, N = int(shape.integers(3, 7)), int(shape.integers(3, 6))
        mesh = tl.TreeMesh((-10.0, -10.0), (10.0, 10.0), level)
        ic = tl.IsentropicVortex(float(rng.uniform(1.0, 5.0)), center=tuple(float(c) for c in rng.uniform(-2.0, 2.0, 2)))
        out.append((mesh, N, _state(ic, mesh.node_coordinates(N), eq)))
    return out


def _step_cfl(case):
    return SHOCK_CFL if case["kind"] in ("riemann", "blast") else _cfl(case["N"])


def _semi(case, seed):
    kind, N = case["kind"], case["N"]
    eq = tl.CompressibleEulerEquations2D(GAMMA)
    ic = _initial(case, seed)
    td = tl.MDRK() if kind == "mdrk" else tl.LW()
    flux = (tl.FluxHLL if case.get("flux") == "hll" else tl.FluxLaxFriedrichs)(case.get("speed", "naive"))
    vi = tl.VolumeIntegralFR(td)
    if kind in ("riemann", "blast"):
        more = {"reconstruction": tl.MUSCLReconstruction()} if kind == "blast" else {}
        vi = tl.VolumeIntegralFRShockCapturing(tl.IndicatorHennemannGassner(alpha_max=0.5), vi, **more)
    solver = tl.DGSEM(N, flux, vi)
    mesh = _mesh(case)
    if kind == "cavity":
        par = tl.CompressibleNavierStokesDiffusion2D(eq, mu=0.001, Prandtl=0.72,
                                                     gradient_variables=tl.GradientVariablesConservative())
        heat = tl.Adiabatic(lambda x, y, t, e: 0.0)
        wall = tl.BoundaryConditionNavierStokesWall(tl.NoSlip(lambda x, y, t, e: (0.0, 0.0)), heat)
        lid = tl.BoundaryConditionNavierStokesWall(tl.NoSlip(lambda x, y, t, e: (1.0, 0.0)), heat)
        vert, hor = tl.boundary_condition_slip_wall_vertical, tl.boundary_condition_slip_wall_horizontal
        bcs = ({"x_neg": vert, "x_pos": vert, "y_neg": hor, "y_pos": hor},
               {"x_neg": wall, "x_pos": wall, "y_neg": wall, "y_pos": lid})
        return tl.SemidiscretizationHyperbolicParabolic(mesh, td, (eq, par), ic, solver, boundary_conditions=bcs)
    more = {"boundary_conditions": tl.BoundaryConditionDirichlet(ic)} if kind == "riemann" else {}
    return tl.SemidiscretizationHyperbolic(mesh, td, eq, ic, solver, **more)


def prepare(case, seed):
    if case["kind"] == "batch":
        b = tl.LWBatch(tl.CompressibleEulerEquations2D(GAMMA))
        insts = _instances(case, seed)
        for mesh, N, _ in insts:
            b.add(mesh, N)
        b.finalize()
        us = [torch.from_numpy(u).cuda() for _, _, u in insts]
        torch.cuda.synchronize()
        return {"case": case, "batch": b, "u0": us, "out": [torch.empty_like(u) for u in us],
                "cfl": [_cfl(N) for _, N, _ in insts]}
    semi = _semi(case, seed)
    u0 = semi.compute_coefficients(0.0)
    state = {"case": case, "semi": semi, "cfl": _step_cfl(case)}
    if case["kind"] == "rhs":
        semi.cache["dt"][0] = semi.max_dt(u0, state["cfl"])
        return state | {"u0": u0, "out": np.empty_like(u0)}
    if case["kind"] == "gradient":
        target = u0.reshape(-1, 4)[:, 0] * (1.0 + 0.05 * np.random.default_rng(seed + 1).standard_normal(u0.size // 4))
        return state | {"u0": torch.from_numpy(u0).cuda().requires_grad_(True), "target": torch.from_numpy(target).cuda()}
    semi._prepare_boundaries(0.0, 0.0, 1.0)
    u0 = torch.from_numpy(u0).cuda()
    torch.cuda.synchronize()
    integ = tl.LWIntegrator(tl.semidiscretize(semi, semi.time_discretization, (0.0, 1e9)))
    return state | {"integ": integ, "u0": u0, "out": torch.empty_like(u0)}


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(state):
    case = state["case"]
    L = _lib.lib()
    if case["kind"] == "rhs":
        tl.rhs(state["out"], state["u0"], state["semi"], 0.0)
        return state["out"]
    if case["kind"] == "gradient":
        state["u0"].grad = None
        uT = tl.lw_solve(state["u0"], state["semi"], case["steps"], state["cfl"], case["every"])
        J = 0.5 * (uT.view(-1, 4)[:, 0] - state["target"]).square().sum()
        J.backward()
        return [uT.detach(), state["u0"].grad]
    if case["kind"] == "batch":
        b, t = state["batch"], ctypes.c_double()
        for i, (u, cfl) in enumerate(zip(state["u0"], state["cfl"])):
            _lib.check(b.ptr, L.tlw_batch_set_state(b.ptr, i, _ptr(u), _lib.TLW_WHERE_DEVICE, 0.0, cfl, 1e9), batch=True)
        b.step(case["steps"])
        for i, u in enumerate(state["out"]):
            _lib.check(b.ptr, L.tlw_batch_get_state(b.ptr, i, _ptr(u), _lib.TLW_WHERE_DEVICE, ctypes.byref(t), None),
                       batch=True)
        return state["out"]
    h, integ = state["semi"].handle, state["integ"]
    _lib.check(h, L.tlw_set_state(h, _ptr(state["u0"]), _lib.TLW_WHERE_DEVICE, 0.0))
    integ.step(case["steps"], state["cfl"])
    t = integ.sync_time()
    _lib.check(h, L.tlw_get_state(h, _ptr(state["out"]), _lib.TLW_WHERE_DEVICE, None))
    return [state["out"], t]


# ---- the least a pass does -----------------------------------------------------------------------------------------
def _flops_per_node(N):
    """Flux pairs, line contractions and stage updates of a Lax-Wendroff step, a multiply-add as two."""
    n = N + 1
    return 80 * n + 589 if N >= 4 else 64 * n + 387


def work(case):
    kind = case["kind"]
    if kind == "batch":
        shape = np.random.default_rng(case["count"])
        nodes = flops = 0
        for _ in range(case["count"]):
            level, N = int(shape.integers(3, 7)), int(shape.integers(3, 6))
            nodes += 4 ** level * (N + 1) ** 2
            flops += 4 ** level * (N + 1) ** 2 * _flops_per_node(N)
        return {"bytes": 64.0 * nodes * case["steps"], "flops": float(flops * case["steps"])}
    n = case["N"] + 1
    if kind in ("warped", "blast", "cavity"):
        elements, per = case["nx"] * case["ny"], 64 + 40        # with the metric terms
    else:
        elements, per = 4 ** case["level"], 64
        if kind == "amr":
            m = 2 ** case["level"]
            inside = sum(1 for k in range(m) if abs(-10.0 + (k + 0.5) * 20.0 / m) <= 4.0)
            elements += 3 * inside * inside
    nodes = elements * n * n
    steps = case.get("steps", 1)
    flops = _flops_per_node(case["N"])
    if kind == "mdrk":
        flops = 64 * n + 410                                      # two stages of two contractions and five flux pairs
    if kind == "gradient":
        per, flops = 3 * per, 3 * flops                           # forward, and a reverse step of twice its work
    return {"bytes": float(per * nodes * steps), "flops": float(flops * nodes * steps)}


# ---- the same in plain torch ---------------------------------------------------------------------------------------
def _basis(N):
    """GLL nodes and weights, the derivative matrix and -M^-1 D^T M, from the Legendre polynomials."""
    P = np.polynomial.legendre.Legendre.basis(N)
    x = np.concatenate([[-1.0], np.sort(P.deriv().roots().real), [1.0]])
    for _ in range(3):                                            # Newton on P_N' at the inner nodes
        x[1:-1] -= P.deriv()(x[1:-1]) / P.deriv(2)(x[1:-1])
    w = 2.0 / (N * (N + 1) * P(x) ** 2)
    d = x[:, None] - x[None, :] + np.eye(N + 1)
    b = 1.0 / d.prod(axis=1)
    D = b[None, :] / b[:, None] / d * (1 - np.eye(N + 1))
    D -= np.diag(D.sum(axis=1))
    return x, w, D, -(D.T * w[None, :]) / w[:, None]


def _interpolation(x, at):
    """[len(at), len(x)]: the Lagrange polynomials of x at the points `at`."""
    return np.array([[np.prod([(t - x[k]) / (x[j] - x[k]) for k in range(len(x)) if k != j]) for j in range(len(x))]
                     for t in at])


def _fluxes(u):
    r, a, b, e = u.unbind(-1)
    v, w = a / r, b / r
    p = (GAMMA - 1.0) * (e - 0.5 * (a * v + b * w))
    return torch.stack([a, a * v + p, a * w, (e + p) * v], -1), torch.stack([b, b * v, b * w + p, (e + p) * w], -1)


def _speeds(u):
    r, a, b, e = u.unbind(-1)
    c = torch.sqrt(GAMMA * (GAMMA - 1.0) * (e - 0.5 * (a * a + b * b) / r) / r)
    return a / r, b / r, c


def _lambda(ul, ur, nx, ny, speed):
    (al, bl, cl), (ar, br, cr) = _speeds(ul), _speeds(ur)
    s = (nx * nx + ny * ny) ** 0.5
    vl, vr = (al * nx + bl * ny).abs(), (ar * nx + br * ny).abs()
    return torch.maximum(vl, vr) + torch.maximum(cl, cr) * s if speed == "naive" else torch.maximum(vl + cl * s, vr + cr * s)


class _Plain:
    """The schemes on [element, j, i, variable] tensors."""

    def __init__(self, case, mesh, N, device):
        self.case, self.N, self.n = case, N, N + 1
        self.speed, self.hll = case.get("speed", "naive"), case.get("flux") == "hll"
        self.shock = case["kind"] == "riemann"
        x, w, D, Dhat = _basis(N)
        self.t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=device)
        self.x, self.w, self.D, self.Dhat = x, w, self.t(D), self.t(Dhat)
        self.metrics = None
        self.mortars, self.boundaries = [], []
        if case["kind"] == "warped":
            self._curved(mesh)
        else:
            self._tree(mesh)

    def _tree(self, mesh):
        self.ij = self.t(mesh.inverse_jacobian).view(-1, 1, 1, 1)
        ids, ors = np.asarray(mesh.interface_neighbor_ids).reshape(-1, 2) - 1, np.asarray(mesh.interface_orientations)
        self.faces = [(o, self.t(ids[ors == o, 0]), self.t(ids[ors == o, 1])) for o in (1, 2)]
        if getattr(mesh, "n_mortars", 0):
            m = np.asarray(mesh.mortar_neighbor_ids).reshape(-1, 3) - 1
            side, mo = np.asarray(mesh.mortar_large_sides), np.asarray(mesh.mortar_orientations)
            for o in (1, 2):
                for s in (1, 2):
                    at = (mo == o) & (side == s)
                    if at.any():
                        self.mortars.append((o, s, *(self.t(m[at, k]) for k in range(3))))
            g, wg = np.polynomial.legendre.leggauss(self.n)
            lg = _interpolation(self.x, g)
            mass = (lg * wg[:, None]).T @ lg
            self.halves = []
            for shift in (-1.0, 1.0):
                to = _interpolation(self.x, 0.5 * (self.x + shift))
                back = np.linalg.solve(mass, 0.5 * (_interpolation(self.x, 0.5 * (g + shift)) * wg[:, None]).T @ lg)
                self.halves.append((self.t(to), self.t(back)))
        if mesh.n_boundaries:
            last = 0
            for d, c in enumerate(mesh.n_boundaries_per_direction):
                self.boundaries.append((d, self.t(np.asarray(mesh.boundary_neighbor_ids)[last:last + c] - 1)))
                last += c

    def _curved(self, mesh):
        X, Y = (self.t(np.transpose(c, (2, 1, 0))) for c in mesh.node_coordinates(self.N))
        dx = lambda a: torch.einsum("ik,ejk->eji", self.D, a)  # noqa: E731
        dy = lambda a: torch.einsum("jk,eki->eji", self.D, a)  # noqa: E731
        self.metrics = [dy(Y), -dy(X), -dx(Y), dx(X)]
        self.ij = (1.0 / (dx(X) * dy(Y) - dy(X) * dx(Y))).unsqueeze(-1)
        nx, ny = mesh.cells
        e = np.arange(nx * ny).reshape(ny, nx)
        # (orientation, left element, right element): the right one's face is the primary
        self.faces = [(1, self.t(np.roll(e, 1, 1).reshape(-1)), self.t(e.reshape(-1))),
                      (2, self.t(np.roll(e, 1, 0).reshape(-1)), self.t(e.reshape(-1)))]

    def contract(self, M, f, g):
        if self.metrics is not None:
            a, b, c, d = (m.unsqueeze(-1) for m in self.metrics)
            f, g = a * f + b * g, c * f + d * g
        return torch.einsum("ik,ejkv->ejiv", M, f) + torch.einsum("jk,ekiv->ejiv", M, g)

    def averages(self, u, dt):
        """The time averages U, F, G of a Lax-Wendroff step."""
        f0, g0 = _fluxes(u)
        U, F, G, f, g = u, f0, g0, f0, g0
        p = {k: u for k in (2, 1, -1, -2)}
        first = {2: -1.0 / 12, 1: 8.0 / 12, -1: -8.0 / 12, -2: 1.0 / 12}
        second = ({2: -1.0 / 12, 1: 16.0 / 12, 0: -30.0 / 12, -1: 16.0 / 12, -2: -1.0 / 12} if self.N >= 4
                  else {1: 1.0, 0: -2.0, -1: 1.0})
        third = {2: 0.5, 1: -1.0, -1: 1.0, -2: -0.5}
        fourth = {2: 0.5, 1: -2.0, 0: 3.0, -1: -2.0, -2: 0.5}    # the scheme's factor 1/2
        fact = 1.0
        for m, stencil in enumerate([first, second, third, fourth][:min(self.N, 4)], 1):
            d = -dt * self.ij * self.contract(self.D, f, g)
            fact *= m
            U = U + d / (fact * (m + 1))
            p = {k: v + d * (float(k) ** m / fact) for k, v in p.items()}
            f = g = 0.0
            for k, c in stencil.items():
                a, b = (f0, g0) if k == 0 else _fluxes(p[k])
                f, g = f + c * a, g + c * b
            F, G = F + f / (fact * (m + 1)), G + g / (fact * (m + 1))
        return U, F, G

    def surface_flux(self, fl, fr, Ul, Ur, ul, ur, nx, ny):
        """f(f_ll, f_rr, a, a', b, b'): Rusanov's speed from a and jump in b, HLL's speeds from b and jump in a."""
        if not self.hll:
            return 0.5 * (fl + fr) - 0.5 * _lambda(Ul, Ur, nx, ny, self.speed).unsqueeze(-1) * (ur - ul)
        (al, bl, cl), (ar, br, cr) = _speeds(ul), _speeds(ur)
        lo, hi = (al * nx + bl * ny - cl).unsqueeze(-1), (ar * nx + br * ny + cr).unsqueeze(-1)
        mid = (hi * fl - lo * fr + lo * hi * (Ur - Ul)) / (hi - lo)
        return torch.where((lo >= 0) & (hi >= 0), fl, torch.where((lo <= 0) & (hi <= 0), fr, mid))

    @staticmethod
    def face(a, o, last):
        at = -1 if last else 0
        return a[:, :, at] if o == 1 else a[:, at]

    def surface(self, du, u, U, F, G, dt, sub=None, boundary=None, scale=1.0):
        """du and the surface integral of the faces' numerical fluxes, without the Jacobian."""
        du = du.clone()
        wf, wl = self.w[0], self.w[-1]
        for o, l, r in self.faces:
            H = F if o == 1 else G
            nx, ny = (1.0, 0.0) if o == 1 else (0.0, 1.0)
            ul, ur = self.face(u, o, True)[l], self.face(u, o, False)[r]
            Ul, Ur = self.face(U, o, True)[l], self.face(U, o, False)[r]
            fl, fr = self.face(H, o, True)[l], self.face(H, o, False)[r]
            if self.metrics is not None:
                # the normal is the right element's, outward (negative); speeds from u, jump in U
                nx, ny = (-self.face(self.metrics[2 * o - 2 + k].unsqueeze(-1), o, False)[r][..., 0] for k in (0, 1))
                Fn = -self.surface_flux(-fr, -fl, ur, ul, Ur, Ul, nx, ny)
            else:
                Fn = self.surface_flux(fl, fr, Ul, Ur, ul, ur, nx, ny)
            if sub is not None:
                Fn = self.blend(Fn, o, l, r, ul, ur, dt, sub)
            self.face(du, o, True).index_add_(0, l, Fn / wl)
            self.face(du, o, False).index_add_(0, r, Fn / -wf)
        for o, s, lower, upper, large in self.mortars:
            H = F if o == 1 else G
            nx, ny = (1.0, 0.0) if o == 1 else (0.0, 1.0)
            big = s == 1                                         # the large element is the left one
            back = 0.0
            for e, (to, proj) in zip((lower, upper), self.halves):
                up = lambda a: torch.einsum("lk,ekv->elv", to, self.face(a, o, big)[large])  # noqa: E731
                own = lambda a: self.face(a, o, not big)[e]  # noqa: E731
                sides = [(up(a), own(a)) if big else (own(a), up(a)) for a in (H, U, u)]
                Fn = self.surface_flux(*sides[0], *sides[1], *sides[2], nx, ny)
                self.face(du, o, not big).index_add_(0, e, Fn / (-wf if big else wl))
                back = back + torch.einsum("lk,ekv->elv", proj, Fn)
            self.face(du, o, big).index_add_(0, large, back / (wl if big else -wf))
        for d, e in self.boundaries:
            o, last = (1 if d < 2 else 2), d % 2 == 1
            ub = self.face(boundary, o, last)[e]
            fb = scale * _fluxes(ub)[o - 1]
            inner = [self.face(a, o, last)[e] for a in (F if o == 1 else G, U, u)]
            pairs = [(a, b) if last else (b, a) for a, b in zip(inner, (fb, scale * ub, ub))]
            Fn = self.surface_flux(*pairs[0], *pairs[1], *pairs[2], 2.0 - o, o - 1.0)
            self.face(du, o, last).index_add_(0, e, Fn / (wl if last else -wf))
        return du

    # shock capturing: the indicator, first-order subcells, and the blended interface flux
    def alpha(self, u):
        n = self.n
        V = np.stack([np.polynomial.legendre.Legendre.basis(m)(self.x) * math.sqrt(m + 0.5) for m in range(n)], 1)
        Vi = self.t(np.linalg.inv(V))
        ind = (GAMMA - 1.0) * (u[..., 0] * u[..., 3] - 0.5 * (u[..., 1] ** 2 + u[..., 2] ** 2))
        m2 = torch.einsum("ai,bj,eji->eba", Vi, Vi, ind) ** 2
        tot, c1, c2 = (m2[:, :k, :k].sum((1, 2)) for k in (n, n - 1, n - 2))
        energy = torch.maximum((tot - c1) / tot, (c1 - c2) / c1)
        thr = 0.5 * 10.0 ** (-1.8 * n ** 0.25)
        raw = 1.0 / (1.0 + torch.exp(-math.log(0.9999 / 0.0001) / thr * (energy - thr)))
        raw = torch.where(raw < 0.001, 0.0, torch.where(raw > 0.999, 1.0, raw)).clamp(max=0.5)
        a = raw.clone()
        for _, l, r in self.faces:
            a.scatter_reduce_(0, l, 0.5 * raw[r], "amax")
            a.scatter_reduce_(0, r, 0.5 * raw[l], "amax")
        return a

    def subcells(self, u):
        """The subcell fluxes between a row's (column's) nodes and what they give the nodes."""
        f, g = _fluxes(u)
        w = self.t(self.w)
        lx = _lambda(u[:, :, :-1], u[:, :, 1:], 1.0, 0.0, self.speed).unsqueeze(-1)
        ly = _lambda(u[:, :-1], u[:, 1:], 0.0, 1.0, self.speed).unsqueeze(-1)
        fx = 0.5 * (f[:, :, :-1] + f[:, :, 1:]) - 0.5 * lx * (u[:, :, 1:] - u[:, :, :-1])
        gy = 0.5 * (g[:, :-1] + g[:, 1:]) - 0.5 * ly * (u[:, 1:] - u[:, :-1])
        dx = torch.nn.functional.pad(fx, (0, 0, 0, 1)) - torch.nn.functional.pad(fx, (0, 0, 1, 0))
        dy = torch.nn.functional.pad(gy, (0, 0, 0, 0, 0, 1)) - torch.nn.functional.pad(gy, (0, 0, 0, 0, 1, 0))
        return fx, gy, dx / w.view(1, 1, -1, 1) + dy / w.view(1, -1, 1, 1)

    def blend(self, Fn, o, l, r, ul, ur, dt, sub):
        a, fx, gy = sub
        nx, ny = 2.0 - o, o - 1.0
        fn = 0.5 * (_fluxes(ul)[o - 1] + _fluxes(ur)[o - 1]) - 0.5 * _lambda(ul, ur, nx, ny, self.speed).unsqueeze(-1) * (ur - ul)
        fil, fir = (self.face(fx if o == 1 else gy, o, s)[e] for e, s in ((l, True), (r, False)))
        alp = (0.5 * (a[l] + a[r])).view(-1, 1, 1).expand(-1, self.n, 1)
        Fb = (1.0 - alp) * Fn + alp * fn
        c = dt * self.ij[0, 0, 0, 0] * 2.0
        good = True
        for low in (ul - c / self.w[-1] * (Fb - fil), ur - c / self.w[0] * (fir - Fb)):
            p = low[..., 3] - 0.5 * (low[..., 1] ** 2 + low[..., 2] ** 2) / low[..., 0]
            good = (low[..., 0] > 0) & (p > 0) & good
        alp = torch.where(good.unsqueeze(-1), alp, 1.0)
        return alp * fn + (1.0 - alp) * Fn

    def rhs(self, u, dt, boundary=None):
        U, F, G = self.averages(u, dt)
        return self.rhs_from(u, U, F, G, dt, boundary)

    def rhs_from(self, u, U, F, G, dt, boundary=None, scale=1.0):
        du = self.contract(self.Dhat, F, G)
        if self.metrics is not None:
            a, b, c, d = (m.unsqueeze(-1) for m in self.metrics)
            F, G = a * F + b * G, c * F + d * G
        sub = None
        if self.shock:
            a = self.alpha(u)
            fx, gy, fv = self.subcells(u)
            e = a.view(-1, 1, 1, 1)
            du, sub = (1.0 - e) * du + e * fv, (a, fx, gy)
        return -self.ij * self.surface(du, u, U, F, G, dt, sub, boundary, scale)

    def first(self, u, dt):
        """u_t dt and the four-point f_t dt, g_t dt of the two-stage scheme."""
        f0, g0 = _fluxes(u)
        d = -dt * self.ij * self.contract(self.D, f0, g0)
        ft = gt = 0.0
        for k, c in ((2, -1.0), (1, 8.0), (-1, -8.0), (-2, 1.0)):
            f, g = _fluxes(u + k * d)
            ft, gt = ft + c / 12 * f, gt + c / 12 * g
        return f0, g0, d, ft, gt

    def step(self, u, dt, boundary=None):
        if self.case["kind"] != "mdrk":
            return u + dt * self.rhs(u, dt, boundary)
        f, g, d, ft, gt = self.first(u, dt)
        us = u + dt * self.rhs_from(u, u / 2 + d / 8, f / 2 + ft / 8, g / 2 + gt / 8, dt)
        _, _, ds, fs, gs = self.first(us, dt)
        return u + dt * self.rhs_from(u, u + d / 6 + ds / 3, f + ft / 6 + fs / 3, g + gt / 6 + gs / 3, dt)

    def dt(self, u, cfl):
        v, w, c = _speeds(u.detach())
        l1, l2 = v.abs() + c, w.abs() + c
        if self.metrics is not None:
            a, b, p, q = self.metrics
            s = self.ij[..., 0].abs()
            l1, l2, ij = (a * l1 + b * l2).abs() * s, (p * l1 + q * l2).abs() * s, 1.0
        else:
            ij = self.ij.view(-1)
        return float(cfl * 2.0 / (self.n * (ij * (l1.amax((1, 2)) + l2.amax((1, 2)))).max()))


def exact(case, seed):
    if case["kind"] in ("blast", "cavity"):
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"

    def steps(plain, u, cfl, count, boundary=None):
        t = 0.0
        for _ in range(count):
            dt = plain.dt(u, cfl)
            u, t = plain.step(u, dt, boundary), t + dt
        return u, t

    if case["kind"] == "batch":
        out = []
        for mesh, N, u in _instances(case, seed):
            u = torch.as_tensor(u, device=device).view(-1, N + 1, N + 1, 4)
            out.append(steps(_Plain(case, mesh, N, device), u, _cfl(N), case["steps"])[0].reshape(-1))
        return out
    mesh, N = _mesh(case), case["N"]
    xy = mesh.node_coordinates(N) if hasattr(mesh, "node_coordinates") else None
    u0 = _state(_initial(case, seed), xy, tl.CompressibleEulerEquations2D(GAMMA))
    plain = _Plain(case, mesh, N, device)
    u = torch.as_tensor(u0, device=device).view(-1, N + 1, N + 1, 4)
    cfl = _step_cfl(case)
    if case["kind"] == "rhs":
        return plain.rhs(u, plain.dt(u, cfl)).reshape(-1).cpu().numpy()
    if case["kind"] == "gradient":
        target = u0.reshape(-1, 4)[:, 0] * (1.0 + 0.05 * np.random.default_rng(seed + 1).standard_normal(u0.size // 4))
        states, dts = [u], []
        with torch.no_grad():
            for _ in range(case["steps"]):
                dts.append(plain.dt(states[-1], cfl))
                states.append(plain.step(states[-1], dts[-1]))
        g = torch.zeros_like(u)
        g.view(-1, 4)[:, 0] = states[-1].reshape(-1, 4)[:, 0] - torch.as_tensor(target, device=device)
        for v, dt in zip(states[-2::-1], dts[::-1]):
            v = v.detach().requires_grad_(True)
            (g,) = torch.autograd.grad(plain.step(v, dt), v, g)
        return [states[-1].reshape(-1), g.reshape(-1)]
    # the Dirichlet data are the initial state's, held
    u, t = steps(plain, u, cfl, case["steps"], u if case["kind"] == "riemann" else None)
    return [u.reshape(-1), t]
