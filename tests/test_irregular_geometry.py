"""Geometries without sheets, where most voxels belong to irregular groups: the step kernel takes
them as groups once there are many.  Fields bitwise those of the direct kernel, and an ensemble
of such grids no slower than it was with one launch per step."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = 0.95 * 36 / (6 * 220000.0)


def blocks(synth, spec, seed, size, all_serca=True):
    """Random domains in blocks of size^3, SERCA across every face between cytosol and network SR."""
    rng = np.random.default_rng(seed)
    shape = spec["voxels"].shape
    c = rng.integers(0, 4, size=tuple(-(-n // size) for n in shape)).astype(np.uint8)
    v = np.kron(c, np.ones((size,) * 3, dtype=np.uint8))[:shape[0], :shape[1], :shape[2]]
    spec["voxels"] = np.ascontiguousarray(v)
    for b in spec["boundaries"]:
        if b["name"] == "serca":
            b["pairs"] = synth._adjacent_pairs(spec["voxels"], 0, 3)
            if not all_serca:                                # every third, in any order
                b["pairs"] = b["pairs"][rng.permutation(len(b["pairs"]))[:len(b["pairs"]) // 3]]
    return spec


@pytest.mark.parametrize("shape,size,all_serca,o", [
    ((45, 44, 42), 3, True, {}),
    ((41, 39, 45), 2, True, dict(force_dirichlet=True)),
    ((48, 40, 43), 3, False, dict(dt_update_react=3.01 * DT)),
    ((47, 48, 37), 2, True, dict(fixed=[(0, 0), (1, 1), (3, 0)], dt_update_stoch=2.01 * DT)),
    ((34, 52, 49), 5, True, dict(surrogate=True, dt_update_react=3.01 * DT)),
    ((46, 40, 47), 2, True, dict(surrogate=True, dt_update_react=2.01 * DT)),
    ((44, 46, 42), 2, True, dict(species=6)),
])
def test_bitwise(pkg, synth, shape, size, all_serca, o):
    """Five realisations: 400,000 voxels, above the irregular ones from which groups are taken."""
    o, n = dict(o), 5
    spec = blocks(synth, synth.tiny(shape), 7, size, all_serca)
    for k in range(5, o.pop("species", 5)):                  # further fixed-point buffers
        spec["species"] = list(spec["species"]) + ["X%d" % k]
        spec["domain_species"] = {d: dict(v, init=list(v["init"]) + [5.0 if d == "cyt" else 0.0],
                                          buffers=list(v["buffers"]) + (d == "cyt") * [
                                              dict(species=[k, 0], k_on=0.02, k_off=0.1, tot=30.0)])
                                  for d, v in spec["domain_species"].items()}
    spec["fixed_domain_species"] = o.pop("fixed", [])
    surrogate = o.pop("surrogate", False)
    opts = dict(h=6.0, tstop=5.0, seed=3, open_states={"ryr": [0, 1, 2]}, **o)
    got = []
    for kernel in (0, 1):
        sim = pkg.Simulation([spec] * n, [dict(opts, seed=3 + r) for r in range(n)])
        sim.set_kernel(kernel)
        if surrogate:
            sim.set_surrogate(pkg.mlp_init(5), 1e-4)
        sim.advance(24)
        got.append([sim.state(r) for r in range(n)])
        sim.close()
    for r in range(n):
        assert np.isfinite(got[0][r]).all()
        np.testing.assert_array_equal(got[0][r], got[1][r])


def step_us(pkg, specs, steps=60):
    n = len(specs)
    sim = pkg.Simulation(specs, [dict(h=6.0, tstop=50.0, seed=k, open_states={"ryr": [0]}) for k in range(n)])
    sim.advance(steps)
    best = 1e9
    for _ in range(4):
        t = time.perf_counter()
        sim.advance(steps)
        best = min(best, time.perf_counter() - t)
    sim.close()
    return best / steps * 1e6


def test_ensemble_not_slower_than_launch_per_step(pkg, synth):
    """24 grids of 100x100x50: with a launch per step 382 us (blocks of 2) and 283 us (blocks of
    8) per step, where the sheet geometry's step takes 104 us now; 15 % for the timing."""
    n = 24
    ref = step_us(pkg, [synth.spark_model((100, 100, 50)) for _ in range(n)])
    for size, bound in ((2, 1.15 * 382 / 104), (8, 1.15 * 283 / 104)):
        us = step_us(pkg, [blocks(synth, synth.spark_model((100, 100, 50)), 1, size) for _ in range(n)])
        assert us < bound * ref, (size, us, ref)


def test_sheets_in_a_large_batch(pkg, synth):
    """The sheets of a dyad leave 1 % irregular voxels: 64 grids have 320,000 of them, and their step
    costs per grid what 24 grids' does (a quarter more while the batch's count decided)."""
    per = [step_us(pkg, [synth.spark_model((100, 100, 50)) for _ in range(n)]) / n for n in (24, 64)]
    assert per[1] < 1.12 * per[0], per
