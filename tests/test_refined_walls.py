"""Meshes with mortars and boundaries in one surface pass (an element may have both, and a wall's and a mortar's code
share the neighbour list), and the kept CFL maximum of refined and curvilinear meshes where a run ends in an
inadmissible state or has source terms. Against the oracle at the package's 1e-12 relative L2 of the state."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NTH = os.cpu_count() or 1


def rel_l2(a, b):
    a, b = a.reshape(-1, 4), b.reshape(-1, 4)
    return np.linalg.norm(a - b, axis=0) / np.maximum(np.linalg.norm(b, axis=0), 1e-300)


def walled(tl, level, patch):
    """RefinedTreeMesh on [-10, 10]^2 without its periodic connections: faces on the outside become boundaries (grouped
    by direction, as Trixi lists them)."""
    m = tl.RefinedTreeMesh((-10.0, -10.0), (10.0, 10.0), level, patch)
    c, h = m.element_centers, m.element_lengths
    ids = m.interface_neighbor_ids.reshape(-1, 2) - 1
    ax = m.interface_orientations - 1
    keep = c[ids[:, 0], ax] < c[ids[:, 1], ax]
    m.interface_neighbor_ids = np.ascontiguousarray(ids[keep] + 1).reshape(-1)
    m.interface_orientations = np.ascontiguousarray(m.interface_orientations[keep])
    m.n_interfaces = int(keep.sum())
    mid = m.mortar_neighbor_ids.reshape(-1, 3) - 1
    ax = m.mortar_orientations - 1
    keep = (c[mid[:, 2], ax] < c[mid[:, 0], ax]) == (m.mortar_large_sides == 1)
    m.mortar_neighbor_ids = np.ascontiguousarray(mid[keep] + 1).reshape(-1)
    m.mortar_large_sides = np.ascontiguousarray(m.mortar_large_sides[keep])
    m.mortar_orientations = np.ascontiguousarray(m.mortar_orientations[keep])
    m.n_mortars = int(keep.sum())
    sides = [np.nonzero(np.abs(c[:, d // 2] + s * (h / 2 - 10.0)) < 1e-9)[0] for d, s in enumerate((-1, 1, -1, 1))]
    m.n_boundaries_per_direction = np.array([len(s) for s in sides], dtype=np.int64)
    m.boundary_neighbor_ids = np.concatenate(sides).astype(np.int64) + 1
    m.boundary_directions = np.repeat(np.arange(1, 5, dtype=np.int64), m.n_boundaries_per_direction)
    m.boundary_orientations = np.where(m.boundary_directions <= 2, 1, 2).astype(np.int64)
    m.boundary_neighbor_sides = np.where(m.boundary_directions % 2 == 0, 1, 2).astype(np.int64)
    m.n_boundaries = len(m.boundary_neighbor_ids)
    faces = 2 * m.n_interfaces + 3 * m.n_mortars + m.n_boundaries
    assert faces == 4 * m.n_elements and m.n_boundaries > 0 and m.n_mortars > 0

    def boundary_node_coordinates(N):
        xy, out = m.node_coordinates(N), np.empty((2, N + 1, m.n_boundaries))
        for b, (e, d) in enumerate(zip(m.boundary_neighbor_ids - 1, m.boundary_directions)):
            out[:, :, b] = (xy[:, 0, :, e], xy[:, N, :, e], xy[:, :, 0, e], xy[:, :, N, e])[d - 1]
        return out

    m.boundary_node_coordinates = boundary_node_coordinates
    return m


# a refined corner (boundary and mortar faces on one element), and a refined stripe from wall to wall
PATCH = {"corner": (2, ((5.0, 5.0), (10.0, 10.0))), "stripe": (2, ((-10.0, -5.0), (10.0, 0.0)))}


def setup(tl, oracle_mod, mesh, N, td, flux, dirichlet=False):
    eq = tl.CompressibleEulerEquations2D(1.4)
    tdo = tl.LW() if td == "lw" else tl.MDRK()
    ic = tl.IsentropicVortex(4.0, center=(1.0, 1.0), velocity=(0.0, 0.0))
    V, H = tl.boundary_condition_slip_wall_vertical, tl.boundary_condition_slip_wall_horizontal
    D = tl.BoundaryConditionDirichlet(lambda x, y, t, e: ic(x, y, 0.0, e), time_independent=True) if dirichlet else V
    solver = tl.DGSEM(N, tl.FluxHLL() if flux else tl.FluxLaxFriedrichs(), tl.VolumeIntegralFR(tdo))
    semi = tl.SemidiscretizationHyperbolic(mesh, tdo, eq, ic, solver,
                                           boundary_conditions={"x_neg": D, "x_pos": V, "y_neg": H, "y_pos": H})
    o = oracle_mod.Oracle(mesh, N, flux_kind=flux)
    o.set_boundary_kinds(np.repeat(np.array([0 if dirichlet else 1, 1, 2, 2], dtype=np.int32), mesh.n_boundaries_per_direction))
    if dirichlet:
        x, y = mesh.boundary_node_coordinates(N)
        now = np.ascontiguousarray(np.transpose(ic(x, y, 0.0, eq), (1, 0, 2)))
        o.set_boundary_data(np.repeat(now[:, :, None, :], N + 1, axis=2), now)
    return semi, o


@pytest.mark.parametrize("N,patch,td,flux,dirichlet", [(1, "corner", "lw", 0, False), (3, "corner", "lw", 1, False),
                                                       (3, "stripe", "mdrk", 0, False), (4, "corner", "mdrk", 1, False),
                                                       (4, "stripe", "lw", 0, True), (5, "corner", "lw", 0, True),
                                                       (6, "stripe", "lw", 1, False)])
def test_steps_between_walls_on_refined_meshes(oracle_mod, tl, N, patch, td, flux, dirichlet):
    mesh = walled(tl, *PATCH[patch])
    semi, o = setup(tl, oracle_mod, mesh, N, td, flux, dirichlet)
    u = semi.compute_coefficients(0.0)
    semi._prepare_boundaries(0.0, 0.0, 1.0)
    integ = tl.LWIntegrator(tl.semidiscretize(semi, semi.time_discretization, (0.0, 1e9)))
    integ.set_state(u, 0.0)
    ref, t = u.copy(), 0.0
    for count in (1, 4):
        integ.step(count, 0.1)
        integ.sync_time()
        _, t = o.steps(ref, count, 0.1, t, 1e9, kind=0 if td == "lw" else 1, nthreads=NTH)
        assert integ.t == pytest.approx(t, rel=1e-13)
    assert np.all(rel_l2(integ.get_state(), ref) < 1e-12)


@pytest.mark.parametrize("N,td", [(4, "lw"), (3, "mdrk")])
def test_source_terms_on_a_refined_mesh(oracle_mod, tl, N, td):
    """t moves on at the end of a step that keeps its CFL maximum, and the sources read it in between."""
    mesh = tl.RefinedTreeMesh((0.0, 0.0), (2.0, 2.0), 2, ((0.5, 0.5), (1.5, 1.5)))
    tdo = tl.LW() if td == "lw" else tl.MDRK()
    semi = tl.SemidiscretizationHyperbolic(mesh, tdo, tl.CompressibleEulerEquations2D(1.4), tl.initial_condition_convergence_test,
                                           tl.DGSEM(N, tl.flux_lax_friedrichs, tl.VolumeIntegralFR(tdo)),
                                           source_terms=tl.source_terms_convergence_test)
    o = oracle_mod.Oracle(mesh, N)
    o.set_source(1, np.ascontiguousarray(np.transpose(mesh.node_coordinates(N), (3, 2, 1, 0))))
    u = semi.compute_coefficients(0.0)
    integ = tl.LWIntegrator(tl.semidiscretize(semi, tdo, (0.0, 1e9)))
    integ.set_state(u, 0.0)
    ref, t = u.copy(), 0.0
    for count, graph in ((1, True), (2, False), (5, True)):
        integ.step(count, 0.1, use_graph=graph)
        integ.sync_time()
        _, t = o.steps(ref, count, 0.1, t, 1e9, kind=0 if td == "lw" else 1, nthreads=NTH)
        assert integ.t == pytest.approx(t, rel=1e-13)
    assert np.all(rel_l2(integ.get_state(), ref) < 1e-12)


def warp(xi, eta):
    s = 0.5 * np.sin(np.pi * xi) * np.sin(np.pi * eta)
    return 10.0 * xi + s, 10.0 * eta + s


MESHES = {"refined": lambda tl: tl.RefinedTreeMesh((-10.0, -10.0), (10.0, 10.0), 2, ((0.0, 0.0), (5.0, 5.0))),
          "refined walls": lambda tl: walled(tl, *PATCH["corner"]),
          "warped": lambda tl: tl.StructuredMesh((6, 5), warp)}


@pytest.mark.parametrize("kind,N,td,cfl", [("refined", 4, "lw", 2.0), ("refined walls", 3, "lw", 3.0),
                                              ("warped", 4, "lw", 1.9), ("warped", 3, "mdrk", 3.0)])
def test_run_that_ends_in_an_inadmissible_state(oracle_mod, tl, kind, N, td, cfl):
    """The last step of a run says nothing of the state it leaves; the step that would start from it does, and neither
    a new state nor a recorded error is blamed afterwards."""
    mesh = MESHES[kind](tl)
    if "walls" in kind:
        semi, o = setup(tl, oracle_mod, mesh, N, td, 0)
    else:
        tdo = tl.LW() if td == "lw" else tl.MDRK()
        semi = tl.SemidiscretizationHyperbolic(mesh, tdo, tl.CompressibleEulerEquations2D(1.4), tl.IsentropicVortex(5.0),
                                               tl.DGSEM(N, tl.flux_lax_friedrichs, tl.VolumeIntegralFR(tdo)))
        o = oracle_mod.Oracle(mesh, N)
    u = semi.compute_coefficients(0.0)
    ref = u.copy()
    o.steps(ref, 1, cfl, 0.0, 1e9, kind=0 if td == "lw" else 1, nthreads=NTH)
    q = ref.reshape(-1, 4)
    pr = 0.4 * (q[:, 3] - 0.5 * (q[:, 1] ** 2 + q[:, 2] ** 2) / q[:, 0])
    assert (pr * q[:, 0] < 0).any()
    integ = tl.LWIntegrator(tl.semidiscretize(semi, semi.time_discretization, (0.0, 1e9)))
    for stepped_further in (True, False):
        integ.set_state(u, 0.0)
        integ.step(1, cfl)
        integ.sync_time()
        if stepped_further:
            integ.step(1, 0.2)
            with pytest.raises(tl.DomainError):
                integ.sync_time()
    integ.set_state(u, 0.0)
    integ.step(3, 0.1)
    integ.sync_time()
