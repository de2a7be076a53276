"""First-order subcells on the TreeMesh at every degree, on a smooth state with one shocked element: elements that blend
(shared and unshared weights) next to elements that do not, whose subcell fluxes only the surface takes. Against the
oracle: the face-adjacent fluxes at 1e-12 of their maximum, the updated states at 1e-12 relative L2, the bars of the
package's shock-capturing tests."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NTH = os.cpu_count() or 1


def rel_l2(a, b):
    a, b = a.reshape(-1, 4), b.reshape(-1, 4)
    return np.linalg.norm(a - b, axis=0) / np.maximum(np.linalg.norm(b, axis=0), 1e-300)


def state(mesh, N):
    x, y = mesh.node_coordinates(N)                       # [i, j, E]
    rho = 1.0 + 0.01 * np.sin(0.2 * np.pi * x) * np.cos(0.1 * np.pi * y)
    v1, v2 = 0.4 + 0.01 * np.cos(0.1 * np.pi * y), -0.3 + 0.01 * np.sin(0.1 * np.pi * x)
    u = np.stack([rho, rho * v1, rho * v2, 1.0 / 0.4 + 0.5 * rho * (v1 ** 2 + v2 ** 2)], axis=-1)
    u[(N + 1) // 2:, :, 21] *= 1.6                        # a contact and pressure jump inside element 21
    return np.ascontiguousarray(np.transpose(u, (2, 1, 0, 3))).reshape(-1)


def reference(oracle_mod, mesh, N):
    o = oracle_mod.Oracle(mesh, N)
    o.set_shock_capturing(True, 0.5, 0.001, True)
    return o


@pytest.mark.parametrize("N,td", [(N, "lw") for N in range(1, 8)] + [(N, "mdrk") for N in (3, 4, 5)])
def test_blended_and_pure_elements(oracle_mod, tl, N, td):
    from trixilw import _lib
    tdo = tl.LW() if td == "lw" else tl.MDRK()
    mesh = tl.TreeMesh((-10.0, -10.0), (10.0, 10.0), 3, periodicity=True)
    vi = tl.VolumeIntegralFRShockCapturing(tl.IndicatorHennemannGassner(alpha_max=0.5), tl.VolumeIntegralFR(tdo))
    semi = tl.SemidiscretizationHyperbolic(mesh, tdo, tl.CompressibleEulerEquations2D(1.4), tl.IsentropicVortex(5.0),
                                           tl.DGSEM(N, tl.flux_lax_friedrichs, vi))
    u = state(mesh, N)
    o = reference(oracle_mod, mesh, N)
    dt = o.max_dt(u, 0.05)
    semi.cache["dt"][0] = dt
    du, kind = np.empty_like(u), 0 if td == "lw" else 1
    (tl.rhs if td == "lw" else tl.rhs_mdrk1)(du, u, semi, 0.0)
    ref = o.rhs(u, 0.0, dt, kind=kind, nthreads=NTH)
    alpha = o.get(6)
    assert 0 < np.count_nonzero(alpha) < mesh.n_elements + (N == 1)   # (N = 1 blends everywhere)
    assert np.all(rel_l2(u + dt * du, u + dt * ref) < 1e-12)
    fnl = o.get(7)
    np.testing.assert_allclose(semi.get_cache(_lib.TLW_CACHE_FN_LOW), fnl, rtol=0, atol=1e-12 * np.abs(fnl).max())
    integ = tl.LWIntegrator(tl.semidiscretize(semi, tdo, (0.0, 1e9)))
    integ.set_state(u, 0.0)
    integ.step(3, 0.05)
    v = u.copy()
    o.steps(v, 3, 0.05, 0.0, 1e9, kind=kind, nthreads=NTH)
    assert np.all(rel_l2(integ.get_state(), v) < 1e-12)
