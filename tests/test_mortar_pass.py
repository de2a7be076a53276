"""The element-centric surface pass with mortar sides: every degree, both patches of refinement (a block, a single
cell, everything but one cell) and the time steppers that share its CFL maximum, against the oracle at the package's
1e-12 relative L2 of the state."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NTH = os.cpu_count() or 1

BOXES = {"block": (3, ((-4.0, -4.0), (4.0, 4.0))), "cell": (2, ((0.0, 0.0), (4.0, 4.0))),
         "all_but_one": (1, ((-10.0, -10.0), (0.0, 10.0)))}


def rel_l2(a, b):
    a, b = a.reshape(-1, 4), b.reshape(-1, 4)
    return np.linalg.norm(a - b, axis=0) / np.maximum(np.linalg.norm(b, axis=0), 1e-300)


@pytest.mark.parametrize("N,box,td,flux", [(1, "block", "lw", 0), (2, "cell", "lw", 1), (3, "block", "mdrk", 0),
                                           (3, "all_but_one", "lw", 1), (4, "cell", "lw", 0), (5, "block", "lw", 0),
                                           (5, "block", "mdrk", 1), (6, "cell", "lw", 0), (7, "block", "lw", 0)])
def test_steps_on_refined_meshes(oracle_mod, tl, N, box, td, flux):
    level, patch = BOXES[box]
    mesh = tl.RefinedTreeMesh((-10.0, -10.0), (10.0, 10.0), level, patch)
    eq = tl.CompressibleEulerEquations2D(1.4)
    tdo = tl.LW() if td == "lw" else tl.MDRK()
    solver = tl.DGSEM(N, tl.FluxHLL() if flux else tl.FluxLaxFriedrichs(), tl.VolumeIntegralFR(tdo))
    semi = tl.SemidiscretizationHyperbolic(mesh, tdo, eq, tl.IsentropicVortex(3.0), solver)
    u = semi.compute_coefficients(0.0)
    o = oracle_mod.Oracle(mesh, N, flux_kind=flux)
    integ = tl.LWIntegrator(tl.semidiscretize(semi, tdo, (0.0, 1e9)))
    integ.set_state(u, 0.0)
    ref, t = u.copy(), 0.0
    for count in (1, 4):
        integ.step(count, 0.1)
        integ.sync_time()
        _, t = o.steps(ref, count, 0.1, t, 1e9, kind=0 if td == "lw" else 1, nthreads=NTH)
        assert integ.t == pytest.approx(t, rel=1e-13)
    assert np.all(rel_l2(integ.get_state(), ref) < 1e-12)
