"""A launch of the step kernel holds the whole GPU, so a call divides its steps into launches
that other streams can get in between, whatever the size of the batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_launch_stays_short(pkg, synth):
    """4,096 steps of 32 grids of 100x100x50 take about 0.6 s: no launch holds the GPU for more
    than a third of a second (the estimate's limit is 0.1 s)."""
    n, steps = 32, 4096
    spec = synth.spark_model((100, 100, 50))
    sim = pkg.Simulation([spec] * n, [dict(h=6.0, tstop=50.0, seed=k, open_states={"ryr": [0]}) for k in range(n)])
    sim.advance(10)
    before = sim.step_launches()
    sim.advance(steps)
    launches = sim.step_launches() - before
    assert sim.last_ms() / launches < 333.0, (sim.last_ms(), launches)
    assert launches < 40
    sim.close()


def test_small_grids_keep_long_launches(pkg, synth):
    sim = pkg.Simulation(synth.tiny((12, 12, 16)), dict(h=6.0, tstop=50.0, seed=1))
    before = sim.step_launches()
    sim.advance(4096)
    assert sim.step_launches() - before == 1
    sim.close()


def test_fields_do_not_depend_on_the_division(pkg, synth):
    """The same steps in one call and one by one."""
    spec, opts = synth.tiny((13, 12, 18)), dict(h=6.0, tstop=50.0, seed=1, open_states={"ryr": [0, 1]})
    a, b = pkg.Simulation(spec, opts), pkg.Simulation(spec, opts)
    a.advance(50)
    for _ in range(50):
        b.advance(1)
    np.testing.assert_array_equal(a.state(), b.state())
    a.close()
    b.close()
