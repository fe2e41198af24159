"""A new tolerance of the surrogate holds on the direct kernel too, whose steps are replayed from a
graph: the same voxels are rejected, and the same fields follow, as on the step kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_new_tolerance(pkg, synth):
    dt = 0.95 * 36 / (6 * 220000.0)
    spec = synth.tiny((14, 12, 18))
    opts = dict(h=6.0, tstop=50.0, seed=1, open_states={"ryr": [0, 1, 2]}, dt_update_react=4.01 * dt)
    p = pkg.mlp_init(5)
    p[-325:] = (0.05 * np.random.default_rng(43).standard_normal(325)).astype(np.float32)
    got = []
    for kernel in (0, 1):
        sim = pkg.Simulation(spec, opts)
        sim.set_kernel(kernel)
        seen = []
        for tol in (1.0, 1e-9):
            sim.set_surrogate(p, tol)
            sim.advance(64)
            seen.append(sim.surrogate_counts())
        got.append((seen, sim.state()))
        sim.close()
    (a, u), (b, v) = got
    assert a == b
    assert a[0] != a[1]
    np.testing.assert_array_equal(u, v)
