"""The CFL maximum that a TreeMesh step keeps for the next one: chunked, graph-replayed and restarted runs against the
oracle's step loop, at sizes on both sides of the rule that lets the volume kernel form dt, with walls (the surface
pass with boundaries) and with the dt clamped to the final time. u at 1e-12 relative L2 after a dozen steps and t at
1e-13, the bars of the package's multi-step tests."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NTH = os.cpu_count() or 1


def rel_l2(a, b):
    a, b = a.reshape(-1, 4), b.reshape(-1, 4)
    return np.linalg.norm(a - b, axis=0) / np.maximum(np.linalg.norm(b, axis=0), 1e-300)


def make(tl, level, N, td, walls=False):
    eq = tl.CompressibleEulerEquations2D(1.4)
    tdo = tl.LW() if td == "lw" else tl.MDRK()
    mesh = tl.TreeMesh((-10.0, -10.0), (10.0, 10.0), level, periodicity=not walls)
    more = {}
    if walls:
        more["boundary_conditions"] = {"x_neg": tl.boundary_condition_slip_wall_vertical,
                                       "x_pos": tl.boundary_condition_slip_wall_vertical,
                                       "y_neg": tl.boundary_condition_slip_wall_horizontal,
                                       "y_pos": tl.boundary_condition_slip_wall_horizontal}
    # between walls a vortex at rest (the moving one is sucked off the wall until the scheme itself has no root to take)
    ic = tl.IsentropicVortex(5.0, velocity=(0.0, 0.0) if walls else (1.0, 1.0))
    return mesh, tl.SemidiscretizationHyperbolic(mesh, tdo, eq, ic,
                                                 tl.DGSEM(N, tl.flux_lax_friedrichs, tl.VolumeIntegralFR(tdo)), **more)


# 2^level squared elements of (N + 1)^2 nodes; the rule's line is at 1.5 million nodes
@pytest.mark.parametrize("level,N,td,walls", [(1, 3, "lw", False), (3, 4, "lw", False), (3, 5, "mdrk", False),
                                              (4, 2, "lw", False), (4, 3, "lw", True), (4, 4, "mdrk", True),
                                              (8, 3, "lw", False), (8, 4, "lw", False), (8, 4, "mdrk", False)])
def test_chunks_of_steps(oracle_mod, tl, level, N, td, walls):
    mesh, semi = make(tl, level, N, td, walls)
    u = semi.compute_coefficients(0.0)
    o = oracle_mod.Oracle(mesh, N)
    if walls:
        per = mesh.n_boundaries_per_direction
        o.set_boundary_kinds(np.repeat(np.array([1, 1, 2, 2], dtype=np.int32), per))
    integ = tl.LWIntegrator(tl.semidiscretize(semi, semi.time_discretization, (0.0, 1e9)))
    kind = 0 if td == "lw" else 1
    for start in range(2):   # the second run starts from a new state on buffers that hold the first one's maxima
        ref = u * (1.0 + 0.1 * start)
        integ.set_state(ref, 0.0)
        t = 0.0
        for count, graph in ((1, True), (3, True), (2, False), (5, True)):
            integ.step(count, 0.2, use_graph=graph)
            integ.sync_time()
            s, t = o.steps(ref, count, 0.2, t, 1e9, kind=kind, nthreads=NTH)
            assert integ.t == pytest.approx(t, rel=1e-13)
        assert integ.iter == 11
        assert np.all(rel_l2(integ.get_state(), ref) < 1e-12)


@pytest.mark.parametrize("td", ["lw", "mdrk"])
def test_end_time_and_limiter_switch(oracle_mod, tl, td):
    mesh, semi = make(tl, 3, 3, td)
    u = semi.compute_coefficients(0.0)
    o = oracle_mod.Oracle(mesh, 3)
    dt = o.max_dt(u, 0.2)
    t_end = 4.5 * dt
    integ = tl.LWIntegrator(tl.semidiscretize(semi, semi.time_discretization, (0.0, t_end)))
    integ.set_state(u, 0.0)
    integ.step(9, 0.2)       # past the end: the rest are no-ops
    integ.sync_time()
    ref = u.copy()
    s, t = o.steps(ref, 9, 0.2, 0.0, t_end, kind=0 if td == "lw" else 1, nthreads=NTH)
    assert integ.t == t_end == t and integ.iter == s == 5
    assert np.all(rel_l2(integ.get_state(), ref) < 1e-12)
    # the limiter (which leaves the vortex as it is) switches the way the maximum is kept, and back
    from trixilw.limiters import install
    integ.tspan = (0.0, 1e9)
    integ.set_state(u, 0.0)
    ref, t = u.copy(), 0.0
    for lim in ((), (tl.PositivityPreservingLimiterZhangShu((5e-6,), (tl.density,)),), ()):
        install(semi, lim)
        integ.step(3, 0.2)
        integ.sync_time()
        _, t = o.steps(ref, 3, 0.2, t, 1e9, kind=0 if td == "lw" else 1, nthreads=NTH)
        assert integ.t == pytest.approx(t, rel=1e-13)
    assert np.all(rel_l2(integ.get_state(), ref) < 1e-12)


@pytest.mark.parametrize("walls,N,td,cfl", [(True, 3, "lw", 2.5), (True, 4, "mdrk", 7.0), (False, 4, "lw", 3.5)])
def test_run_that_ends_in_an_inadmissible_state(oracle_mod, tl, walls, N, td, cfl):
    """A step far past the stability limit leaves negative pressures. Between walls the step itself is sound and the
    next one, which has no wave speed, is not; a plain periodic mesh reports its new state at once; a recorded run
    never steps from its last state and says nothing of it."""
    mesh, semi = make(tl, 3, N, td, walls)
    u = semi.compute_coefficients(0.0)
    o = oracle_mod.Oracle(mesh, N)
    if walls:
        o.set_boundary_kinds(np.repeat(np.array([1, 1, 2, 2], dtype=np.int32), mesh.n_boundaries_per_direction))
    ref = u.copy()
    o.steps(ref, 1, cfl, 0.0, 1e9, kind=0 if td == "lw" else 1, nthreads=NTH)
    q = ref.reshape(-1, 4)
    pr = 0.4 * (q[:, 3] - 0.5 * (q[:, 1] ** 2 + q[:, 2] ** 2) / q[:, 0])
    assert (pr * q[:, 0] < 0).any()
    integ = tl.LWIntegrator(tl.semidiscretize(semi, semi.time_discretization, (0.0, 1e9)))
    integ.set_state(u, 0.0)
    integ.step(1, cfl)
    if walls:
        integ.sync_time()
        integ.step(1, 0.2)
    with pytest.raises(tl.DomainError):
        integ.sync_time()
    if not walls:
        assert np.isfinite(tl.forward_record(semi, u, 1, cfl, 1)).all()
