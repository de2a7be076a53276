"""Orders of calls on a handle that the library refuses, or that it has to keep consistent."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(tl, N, td="lw", periodic=True):
    tdo = tl.LW() if td == "lw" else tl.MDRK()
    mesh = tl.TreeMesh((-10.0, -10.0), (10.0, 10.0), 3, periodicity=periodic)
    solver = tl.DGSEM(N, tl.flux_lax_friedrichs, tl.VolumeIntegralFR(tdo))
    more = {}
    if not periodic:
        more["boundary_conditions"] = {"x_neg": tl.boundary_condition_slip_wall_vertical,
                                       "x_pos": tl.boundary_condition_slip_wall_vertical,
                                       "y_neg": tl.boundary_condition_slip_wall_horizontal,
                                       "y_pos": tl.boundary_condition_slip_wall_horizontal}
    ic = tl.IsentropicVortex(5.0, velocity=(1.0, 1.0) if periodic else (0.0, 0.0))
    return tl.SemidiscretizationHyperbolic(mesh, tdo, tl.CompressibleEulerEquations2D(1.4), ic, solver, **more)


def test_mortars_after_navier_stokes_are_refused(tl):
    """Nothing is launched: the mesh upload, the Navier-Stokes terms and then the mortars, whose sides no Navier-Stokes
    kernel takes."""
    from trixilw import _lib
    L = _lib.lib()
    semi = make(tl, 3)
    m = tl.RefinedTreeMesh((-10.0, -10.0), (10.0, 10.0), 2, ((0.0, 0.0), (4.0, 4.0)))
    h = semi.handle
    ij = np.ascontiguousarray(m.inverse_jacobian)
    dp = lambda a: a.ctypes.data_as(_lib.ctypes.POINTER(_lib.ctypes.c_double))
    ip = lambda a: a.ctypes.data_as(_lib.ctypes.POINTER(_lib.ctypes.c_int64))
    upload = lambda: _lib.check(h, L.tlw_set_tree_mesh(h, m.n_elements, dp(ij), m.n_interfaces, ip(m.interface_neighbor_ids),
                                                       ip(m.interface_orientations), 0, None, None, None, None))
    mortars = lambda count: L.tlw_set_tree_mortars(h, count, ip(m.mortar_neighbor_ids), ip(m.mortar_large_sides),
                                                   ip(m.mortar_orientations))
    upload()
    _lib.check(h, L.tlw_set_parabolic(h, 1e-3, 0.72))
    assert mortars(m.n_mortars) == _lib.TLW_E_UNSUPPORTED
    assert mortars(0) == _lib.TLW_OK
    upload()                                  # a new mesh has no Navier-Stokes terms
    assert mortars(m.n_mortars) == _lib.TLW_OK
    assert L.tlw_set_parabolic(h, 1e-3, 0.72) == _lib.TLW_E_UNSUPPORTED


@pytest.mark.parametrize("N,td,periodic,limiter", [(3, "lw", True, False), (4, "mdrk", True, False), (4, "lw", False, False),
                                                   (3, "lw", True, True)])
def test_split_steps_between_steps(oracle_mod, tl, N, td, periodic, limiter):
    """On a mesh without halo faces the split step may stand between runs of plain steps, which then take the time step
    of the state it left. dt of every step and the state against the oracle, at the bars of the multi-step tests."""
    from trixilw import _lib
    L = _lib.lib()
    semi = make(tl, N, td, periodic)
    if limiter:   # (leaves the vortex as it is; the steps keep per-element maxima)
        from trixilw.limiters import install
        install(semi, (tl.PositivityPreservingLimiterZhangShu((5e-6,), (tl.density,)),))
    o = oracle_mod.Oracle(semi.mesh, N)
    if not periodic:
        o.set_boundary_kinds(np.repeat(np.array([1, 1, 2, 2], dtype=np.int32), semi.mesh.n_boundaries_per_direction))
    u = semi.compute_coefficients(0.0)
    integ = tl.LWIntegrator(tl.semidiscretize(semi, semi.time_discretization, (0.0, 1e9)))
    integ.set_state(u, 0.0)
    h = semi.handle

    def split(count):
        for _ in range(count):
            _lib.check(h, L.tlw_dd_begin(h, 0.2, 0.0, 1e9))
            for _stage in range(L.tlw_dd_stages(h)):
                _lib.check(h, L.tlw_dd_volume(h))
                _lib.check(h, L.tlw_dd_finish(h))

    ref, t = u.copy(), 0.0
    for run, count in ((lambda c: integ.step(c, 0.2), 3), (split, 3), (lambda c: integ.step(c, 0.2), 2), (split, 2),
                       (lambda c: integ.step(c, 0.2, use_graph=False), 1)):
        run(count)
        integ.sync_time()
        _, t = o.steps(ref, count, 0.2, t, 1e9, kind=0 if td == "lw" else 1)
        assert integ.t == pytest.approx(t, rel=1e-13)
    a, b = integ.get_state().reshape(-1, 4), ref.reshape(-1, 4)
    assert np.all(np.linalg.norm(a - b, axis=0) < 1e-12 * np.linalg.norm(b, axis=0))


def test_recorded_run_after_host_steps(tl):
    """Host-buffer stepping changes the handle's state buffers and leaves its last download in flight; a recorded run
    after it (whose graph was captured before) gives the same state and leaves the download alone."""
    semi = make(tl, 4)
    integ = tl.LWIntegrator(tl.semidiscretize(semi, semi.time_discretization, (0.0, 1e9)))
    u = semi.compute_coefficients(0.0)
    integ.set_state(u, 0.0)
    first = tl.forward_record(semi, u, 7, 0.2, 3)
    a, b, c = (integ.pinned_state() for _ in range(3))
    a[:] = 1.01 * u
    integ.step_host(a, b, 0.0, 2, 0.2)
    integ.synchronize()
    expected = b.copy()
    for _ in range(2):
        integ.step_host(a, c, 0.0, 2, 0.2)
        np.testing.assert_array_equal(tl.forward_record(semi, u, 7, 0.2, 3), first)
        integ.synchronize()
        np.testing.assert_array_equal(c, expected)
