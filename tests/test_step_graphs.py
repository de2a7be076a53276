"""The step graphs of a handle: when the graph of eight steps is captured, and that runs replayed from it are the runs
without graphs, to the bit."""
from collections import Counter

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(tl, td="lw"):
    tdo = tl.LW() if td == "lw" else tl.MDRK()
    mesh = tl.TreeMesh((-10.0, -10.0), (10.0, 10.0), 2)
    semi = tl.SemidiscretizationHyperbolic(mesh, tdo, tl.CompressibleEulerEquations2D(1.4), tl.IsentropicVortex(3.0),
                                           tl.DGSEM(3, tl.flux_lax_friedrichs, tl.VolumeIntegralFR(tdo)))
    integ = tl.LWIntegrator(tl.semidiscretize(semi, tdo, (0.0, 1e9)))
    integ.set_state(semi.compute_coefficients(0.0), 0.0)
    return integ


def graphs_made(call):
    """The graphs instantiated while call() runs (skips where the profiler sees no runtime calls)."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        call()
    seen = Counter(e.name for e in p.events())
    if not seen["cudaGraphLaunch"]:
        pytest.skip("the profiler reports no CUDA runtime calls here")
    return seen["cudaGraphInstantiate"]


def test_eight_step_graph_is_earned_or_hidden(tl):
    """A new handle captures its graphs of one and two steps; the one of eight not for a run whose remaining steps it
    could not take, but behind the queued steps of a long one, or once many short calls have earned it."""
    def step(integ, n):
        integ.step(n, 0.1)
        integ.sync_time()

    a = run(tl)
    assert graphs_made(lambda: step(a, 25)) == 3
    assert graphs_made(lambda: [step(a, 16) for _ in range(5)]) == 0
    assert graphs_made(lambda: step(a, 64)) == 1
    assert graphs_made(lambda: [step(a, n) for n in (64, 16, 9)]) == 0
    b = run(tl)
    assert graphs_made(lambda: step(b, 64)) == 4
    c = run(tl)
    assert graphs_made(lambda: [step(c, 16) for _ in range(40)]) == 4


@pytest.mark.parametrize("td", ["lw", "mdrk"])
def test_replayed_runs_equal_plain_ones(tl, td):
    plain, graphed = run(tl, td), run(tl, td)
    for n in (70, 9, 8, 33, 1, 40):
        plain.step(n, 0.1, use_graph=False)
        graphed.step(n, 0.1)
        plain.sync_time()
        graphed.sync_time()
        assert graphed.t == plain.t and graphed.iter == plain.iter
    np.testing.assert_array_equal(graphed.get_state(), plain.get_state())
