"""The time limit of the step kernel's barrier, reached without a fault: with the hook of
csp_test_wait_timeout armed one CTA leaves without arriving, and the CTAs of its team set the
error when their waits run out.  (That the hook's CTA does not set it itself is read from the
source: otherwise the waits would end by the error word, and their limit would never be met.)"""
import os
import time

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hpc-ca-phospattern_b200", "csrc")


def test_the_hook_sets_no_error_where_others_wait():
    src = open(os.path.join(CSRC, "csp_march.cuh")).read()
    kernel = src[src.index("k_march(const __grid_constant__ MarchArgs A)"):]
    hook = kernel[kernel.index("if (A.inject"):kernel.index("for (int e = A.first[team]")]
    assert "atomicOr" not in hook
    assert "if (!waited_for" in hook


@pytest.mark.gpu
@pytest.mark.parametrize("n,stopped", [(1, False), (5, False), (1, True)])
def test_waits_run_out(pkg, synth, n, stopped):
    """A grid of 60x60x40 has 1,160 units and more than one CTA per team whatever the plan; a
    stopped one has no barrier, and the hook's own wait runs out."""
    dt = 0.95 * 36 / (6 * 220000.0)
    opts = dict(h=6.0, tstop=(4.5 if stopped else 1000) * dt, seed=1, open_states={"ryr": [0]})
    sim = pkg.Simulation([synth.spark_model((60, 60, 40))] * n, [opts] * n)
    sim.advance(6)
    assert sim.lib.csp_test_wait_timeout(sim.h, 1) == 0
    t = time.perf_counter()
    with pytest.raises(pkg.CspError) as e:
        sim.advance(3)
    assert e.value.code == -5 and "bounded wait timed out" in str(e.value)
    assert time.perf_counter() - t < 0.9               # the hook's limit, not the one second of other launches
    sim.close()
    fresh = pkg.Simulation(synth.tiny((12, 12, 16)), dict(h=6.0, tstop=5.0, seed=1))
    fresh.advance(20)
    assert fresh.info().step == 20
    fresh.close()
