"""Rejected network outputs are gathered over a warp's tiles before they are integrated: an
ensemble, whose warps meet several realisations, against each realisation alone (bitwise: a
voxel's increment does not depend on what its warp gathered with it)."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("tensor_cores", [1, 2])
@pytest.mark.parametrize("scale", [0.02, 1.0])          # few and most outputs rejected
def test_rejects_across_realisations(pkg, synth, tensor_cores, scale):
    rng = np.random.default_rng(5)
    params = (scale * pkg.mlp_init(2)).astype(np.float32)
    specs, opts = [], []
    for r, shape in enumerate([(20, 18, 17), (9, 8, 7), (14, 22, 16)]):
        spec = synth.tiny(shape, serca=False, pryr=False)
        spec["boundaries"] = []                          # no gating: the draws depend on the ensemble
        spec.pop("ryr", None)
        specs.append(spec)
        opts.append(dict(h=6.0, tstop=1.0, seed=3, dt_update_react=10 * 0.95 * 36 / (6 * 220000.0)))
    alone, states = [], []
    for spec, o in zip(specs, opts):
        sim = pkg.Simulation(spec, o)
        u = sim.state() * rng.uniform(0.3, 1.0, sim.state().shape)
        sim.set_state(u)
        states.append(u)
        sim.set_surrogate(params, 1e-4)
        sim.set_surrogate_tensor_cores(tensor_cores)
        sim.advance(20)
        alone.append((sim.state(), sim.surrogate_counts()))
        sim.close()
    sim = pkg.Simulation(specs, opts)
    for r, u in enumerate(states):
        sim.set_state(u, r)
    sim.set_surrogate(params, 1e-4)
    sim.set_surrogate_tensor_cores(tensor_cores)
    sim.advance(20)
    for r, (u, _) in enumerate(alone):
        np.testing.assert_array_equal(sim.state(r), u)
    counts = sim.surrogate_counts()
    np.testing.assert_array_equal(counts, np.sum([c for _, c in alone], axis=0))
    assert counts[1] > 0 and counts[2] > 0
    sim.close()
