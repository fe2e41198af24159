"""The output path's kernels against the same sums over the downloaded state: rows that are no
multiple of four voxels, a row longer than a warp takes at once, domains without voxels, a
snapshot large enough for several host threads.

Tolerances: minima and maxima are values of the state (equal); sums of n <= 3e5 FP64 terms
differ by their order, n * 1.1e-16 relative at most (all terms are positive)."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(6, 6, 6), (9, 7, 19), (12, 6, 301), (70, 64, 66)])
def test_outputs_against_state(pkg, synth, shape):
    spec = synth.tiny(shape)
    opts = dict(h=6.0, tstop=1.0, seed=4, open_states={"ryr": [0]})
    sim = pkg.Simulation(spec, opts)
    sim.advance(11)
    u = sim.state()
    sim.snapshot_async()
    np.testing.assert_array_equal(sim.snapshot_wait(), u)
    mn, mx, tot, opened = sim.outputs()
    dom = np.asarray(spec["voxels"])
    h = sim.info().h
    f32 = np.finfo(np.float32)
    rtol = 1.2e-16 * u[0].size + 1e-14
    for d in range(mn.shape[0]):
        for s in range(u.shape[0]):
            v = u[s][dom == d]
            assert mn[d, s] == (min(v.min(), f32.max) if v.size else f32.max)
            assert mx[d, s] == (max(v.max(), f32.tiny) if v.size else f32.tiny)
            np.testing.assert_allclose(tot[d, s], v.sum() * h**3 if v.size else 0.0, rtol=rtol)
    inf = sim.info()
    states = [sim.channels(b) for b, d in enumerate(spec["boundaries"]) if inf.num_channels[b]]
    np.testing.assert_array_equal(opened, np.concatenate(states))
    conv, offsets = [2.0e3, 3.0e3, 5.0e3], [0.5 * n * h for n in shape]
    x = [np.arange(n) * h for n in shape]

    def gauss(t, c):
        return np.exp(-t * t / 2 / c) / np.sqrt(2 * np.pi * c)

    for axis in range(3):
        w = [np.ones(n) if a == axis else gauss(offsets[a] - x[a], conv[a]) for a, n in enumerate(shape)]
        plane = np.einsum("xyz,x,y,z->" + "xyz"[axis], u[1], *w)
        want = gauss(x[axis][:, None] - x[axis][None, :], conv[axis]) @ plane
        np.testing.assert_allclose(sim.linescan(1, axis, offsets, conv), want, rtol=rtol)
    sim.close()
