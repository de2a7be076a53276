"""Volume kernels on meshes whose element count is no multiple of the elements per CTA (partly filled last CTA, odd
sides) at every degree: the plane layouts, the whole-element warps of N = 3 and the per-node stencil sums differ by
degree. GPU against the oracle; the bar is the package's 1e-12 relative L2 of u + dt du (a few hundred operations of
1.1e-16 each a node; du itself, which cancels, at 1e-11)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NTH = os.cpu_count() or 1


def rel_l2(a, b):
    a, b = a.reshape(-1, 4), b.reshape(-1, 4)
    return np.linalg.norm(a - b, axis=0) / np.maximum(np.linalg.norm(b, axis=0), 1e-300)


def make(tl, mesh, N, td):
    eq = tl.CompressibleEulerEquations2D(1.4)
    tdo = tl.LW() if td == "lw" else tl.MDRK()
    return tl.SemidiscretizationHyperbolic(mesh, tdo, eq, tl.IsentropicVortex(5.0),
                                           tl.DGSEM(N, tl.flux_lax_friedrichs, tl.VolumeIntegralFR(tdo)))


def warp(xi, eta):
    x, y = 10.0 * xi, 10.0 * eta
    s = np.sin(np.pi * xi) * np.sin(np.pi * eta)
    return x + s, y + s


@pytest.mark.parametrize("td,N", [("lw", N) for N in range(1, 8)] + [("mdrk", N) for N in range(3, 8)])
def test_tree_with_a_refined_cell(oracle_mod, tl, td, N):
    # 19 elements: 15 coarse ones and the four children of one
    mesh = tl.RefinedTreeMesh((-10.0, -10.0), (10.0, 10.0), 2, ((0.0, 0.0), (4.0, 4.0)))
    assert mesh.n_elements == 19
    semi = make(tl, mesh, N, td)
    u = semi.compute_coefficients(0.0)
    o = oracle_mod.Oracle(mesh, N)
    dt = o.max_dt(u, 0.3)
    semi.cache["dt"][0] = dt
    du = np.empty_like(u)
    (tl.rhs if td == "lw" else tl.rhs_mdrk1)(du, u, semi, 0.0)
    ref = o.rhs(u, 0.0, dt, kind=0 if td == "lw" else 1)
    assert np.all(rel_l2(u + dt * du, u + dt * ref) < 1e-12)
    assert np.all(rel_l2(du, ref) < 1e-11)
    if td == "mdrk":
        us = u + dt * ref
        tl.rhs_mdrk2(du, u, semi, 0.0, us)
        ref = o.rhs(u, 0.0, dt, kind=2, us=us)
        assert np.all(rel_l2(u + dt * du, u + dt * ref) < 1e-12)


@pytest.mark.parametrize("N", range(3, 8))
@pytest.mark.parametrize("cells", [(7, 3), (13, 11)])
def test_warped_steps_on_odd_sides(oracle_mod, tl, N, cells):
    mesh = tl.StructuredMesh(cells, warp)
    semi = make(tl, mesh, N, "lw")
    u = semi.compute_coefficients(0.0)
    integ = tl.LWIntegrator(tl.semidiscretize(semi, semi.time_discretization, (0.0, 1e9)))
    integ.set_state(u, 0.0)
    integ.step(3, 0.2)
    integ.sync_time()
    ref = u.copy()
    _, t = oracle_mod.Oracle(mesh, N).steps(ref, 3, 0.2, 0.0, 1e9, nthreads=NTH)
    assert integ.t == pytest.approx(t, rel=1e-13)
    assert np.all(rel_l2(integ.get_state(), ref) < 1e-12)
