"""The element-centric surface pass of curvilinear meshes where they can go wrong: meshes
one cell wide (an element is its own neighbour), odd sides, turned element frames (reversed faces, primary and
secondary in every combination), MDRK. Steps against the oracle at 1e-12 relative L2 of the state; the
walled and Navier-Stokes forms are held by the wall and parabolic tests."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NTH = os.cpu_count() or 1


def rel_l2(a, b):
    a, b = a.reshape(-1, 4), b.reshape(-1, 4)
    return np.linalg.norm(a - b, axis=0) / np.maximum(np.linalg.norm(b, axis=0), 1e-300)


def warp(xi, eta):
    x, y = 10.0 * xi, 10.0 * eta
    s = 0.5 * np.sin(np.pi * xi) * np.sin(np.pi * eta)
    return x + s, y + s


@pytest.mark.parametrize("N,cells,turned,td,flux", [(3, (1, 5), False, "lw", 0), (3, (5, 1), False, "mdrk", 0),
                                                    (4, (7, 5), True, "lw", 1), (4, (9, 4), True, "mdrk", 0),
                                                    (5, (3, 3), True, "lw", 0), (6, (5, 3), True, "lw", 0),
                                                    (7, (2, 3), True, "lw", 1)])
def test_steps(oracle_mod, tl, N, cells, turned, td, flux):
    mesh = tl.StructuredMesh(cells, warp)
    u = None
    eq = tl.CompressibleEulerEquations2D(1.4)
    if turned:
        mesh = tl.rotate_elements(mesh.curved(N), np.random.default_rng(N).integers(0, 4, cells[0] * cells[1]))
    tdo = tl.LW() if td == "lw" else tl.MDRK()
    solver = tl.DGSEM(N, tl.FluxHLL() if flux else tl.FluxLaxFriedrichs(), tl.VolumeIntegralFR(tdo))
    semi = tl.SemidiscretizationHyperbolic(mesh, tdo, eq, tl.IsentropicVortex(2.0), solver)
    u = semi.compute_coefficients(0.0)
    integ = tl.LWIntegrator(tl.semidiscretize(semi, tdo, (0.0, 1e9)))
    integ.set_state(u, 0.0)
    o = oracle_mod.Oracle(mesh, N, flux_kind=flux)
    ref, t = u.copy(), 0.0
    for count in (1, 4):
        integ.step(count, 0.1)
        integ.sync_time()
        _, t = o.steps(ref, count, 0.1, t, 1e9, kind=0 if td == "lw" else 1, nthreads=NTH)
        assert integ.t == pytest.approx(t, rel=1e-13)
    assert np.all(rel_l2(integ.get_state(), ref) < 1e-12)
