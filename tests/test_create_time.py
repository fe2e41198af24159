"""Creating a handle: the boundary voxels are gathered realisation by realisation, so irregular
geometries cost little more host time and memory than the sheets of a dyad."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def create_s(pkg, specs):
    opts = [dict(h=6.0, tstop=50.0, seed=k) for k in range(len(specs))]
    best = 1e9
    for _ in range(3):
        t = time.perf_counter()
        sim = pkg.Simulation(specs, opts)
        best = min(best, time.perf_counter() - t)
        sim.close()
    return best


def test_irregular_geometry(pkg, synth):
    """24 grids of 100x100x50 without fluxes, random domains in blocks of 2^3 against one domain:
    3.1 times as long; 8 times when the whole batch's boundary voxels were gathered in one list."""
    rng = np.random.default_rng(1)
    spec = synth.spark_model((100, 100, 50), serca=False)
    spec["boundaries"] = []
    spec.pop("ryr")
    plain = dict(spec, voxels=np.zeros((100, 100, 50), dtype=np.uint8))
    blocks = np.kron(rng.integers(0, 4, size=(50, 50, 25)), np.ones((2, 2, 2))).astype(np.uint8)
    a = create_s(pkg, [plain] * 24)
    b = create_s(pkg, [dict(spec, voxels=np.ascontiguousarray(blocks))] * 24)
    assert b < 5 * a, (a, b)
