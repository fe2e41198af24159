"""The first call on a batch plans its launch: each realisation's segments are cut once, not once
for every number of teams that the plan looks at."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_long_grids(pkg, synth):
    """40 grids of 900 to 1,290 planes of their own sizes: the plan took 0.42 s."""
    base = synth.tiny((12, 12, 16), serca=False, pryr=False)
    base["boundaries"] = []
    base.pop("ryr")
    specs = [dict(base, voxels=np.zeros((900 + 10 * k, 12, 16), dtype=np.uint8)) for k in range(40)]
    best = 1e9
    for _ in range(2):                                     # (the host may be busy)
        sim = pkg.Simulation(specs, [dict(h=6.0, tstop=1.0, seed=1)] * len(specs))
        t = time.perf_counter()
        sim.advance(1)
        best = min(best, time.perf_counter() - t)
        assert sim.info(39).step == 1
        sim.close()
    assert best < 0.25, best
