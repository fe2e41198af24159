"""The autotuner compares the step kernel and the direct kernel by what a step of a run takes of
each: its figures agree with timed calls, so the choice is between like quantities.  And tuning
leaves no trace in channels, counts or fields."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def step_ms(sim, kernel, steps=512):
    sim.set_kernel(kernel)
    sim.advance(steps)
    best = 1e9
    for _ in range(5):
        t = time.perf_counter()
        sim.advance(steps)
        best = min(best, time.perf_counter() - t)
    return best / steps * 1e3


@pytest.mark.parametrize("sheets", [False, True])
def test_figures_agree_with_calls(pkg, synth, sheets):
    """Before, the direct candidate lacked two of its launches and the step kernel's had a quarter
    of a launch in each step (1.6 of a step for the plain box).  (A candidate far behind is timed
    once, cold, so its figure has no upper bound.)"""
    spec = synth.tiny((24, 24, 24))
    if not sheets:
        spec["voxels"] = np.zeros_like(spec["voxels"])
        spec["boundaries"] = []
        for k in ("ryr", "p_ryr", "serca"):
            spec.pop(k)
    sim = pkg.Simulation(spec, dict(h=6.0, tstop=100.0, seed=1))
    rep = sim.autotune(repeats=20)
    direct = [c["ms"] for c in rep["candidates"] if c["segment"] < 0]
    march = [c["ms"] for c in rep["candidates"] if c["segment"] >= 0]
    assert len(direct) == 1 and rep["chosen"]["segment"] >= 0
    assert 0.7 < direct[0] / step_ms(sim, 1)
    assert 0.7 < min(march) / step_ms(sim, 0) < 1.3
    sim.close()


def test_no_trace(pkg, synth):
    spec = synth.tiny((14, 12, 18))
    opts = dict(h=6.0, tstop=100.0, seed=1, tabort=0.01, open_states={"ryr": [0, 1], "p_ryr": [0]})
    sims = []
    for tuned in (False, True):
        sim = pkg.Simulation([spec, spec], [opts, dict(opts, seed=2)])
        sim.set_kernel(0)
        sim.advance(7)
        if tuned:
            sim.autotune(repeats=3)
            sim.set_kernel(0)
        flags = [sim.advance(60).tolist() for _ in range(12)]
        sims.append((flags, [sim.state(r) for r in range(2)], [sim.channels(b, r) for r in range(2) for b in range(2)],
                     [sim.info(r).step for r in range(2)]))
        sim.close()
    (fa, ua, ca, sa), (fb, ub, cb, sb) = sims
    assert fa == fb and sa == sb
    for x, y in zip(ua + ca, ub + cb):
        np.testing.assert_array_equal(x, y)
