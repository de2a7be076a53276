"""Navier-Stokes steps at the grid sizes where the volume launch asks for more shared memory than it uses: up to one CTA
an SM, up to two, more, and a degree whose own shared memory is the larger. Against the oracle at the package's 1e-12."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NTH = os.cpu_count() or 1


# elements a CTA: N = 3 8, N = 4 5, N = 5 3, N = 7 2; 148 SMs
@pytest.mark.parametrize("N,cells", [(3, (37, 32)), (3, (33, 36)), (4, (20, 37)), (4, (27, 28)), (4, (40, 37)), (4, (41, 37)),
                                     (5, (30, 30)), (7, (12, 12)), (7, (16, 20))])
def test_steps(oracle_mod, tl, N, cells):
    eq = tl.CompressibleEulerEquations2D(1.4)
    par = tl.CompressibleNavierStokesDiffusion2D(eq, mu=0.02, Prandtl=0.72)
    mesh = tl.StructuredMesh(cells, lambda xi, eta: (10.0 * xi + 0.5 * np.sin(np.pi * eta), 10.0 * eta))
    semi = tl.SemidiscretizationHyperbolicParabolic(mesh, tl.LW(), (eq, par), tl.IsentropicVortex(3.0),
                                                    tl.DGSEM(N, tl.flux_lax_friedrichs, tl.VolumeIntegralFR(tl.LW())))
    o = oracle_mod.Oracle(mesh, N)
    o.set_parabolic(0.02, 0.72)
    u = semi.compute_coefficients(0.0)
    integ = tl.LWIntegrator(tl.semidiscretize(semi, tl.LW(), (0.0, 1e9)))
    integ.set_state(u, 0.0)
    integ.step(3, 0.3)
    integ.sync_time()
    ref = u.copy()
    _, t = o.steps(ref, 3, 0.3, 0.0, 1e9, nthreads=NTH)
    assert integ.t == pytest.approx(t, rel=1e-13)
    a, b = integ.get_state().reshape(-1, 4), ref.reshape(-1, 4)
    assert np.all(np.linalg.norm(a - b, axis=0) < 1e-12 * np.linalg.norm(b, axis=0))
