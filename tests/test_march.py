"""The step kernel (kernel 0: whole steps, many to a launch) against the direct kernel, which
computes every voxel with the general per-voxel arithmetic and the fluxes row by row: fields,
channel states and step counts are equal bitwise, for grids at the edges of its units (rows
that are no multiple of 4, planes below, at and above 128 positions, one plane, more columns
than warps), for geometries without any sheet (random domains, random SERCA and channel
pairs), for ensembles with more realisations than are in flight at once, and however the
steps are divided into calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(12, 12, 16), (9, 11, 9), (7, 13, 21), (16, 8, 16), (5, 33, 30), (40, 6, 17), (34, 35, 11), (6, 70, 66)]


def both(pkg, specs, opts, steps, calls=1):
    """The same run on both kernels; returns the (step, direct) simulations."""
    sims = []
    for kernel in (0, 1):
        sim = pkg.Simulation(specs, opts)
        sim.set_kernel(kernel)
        for _ in range(calls if kernel == 0 else 1):
            sim.advance(steps // calls if kernel == 0 else steps)
        sims.append(sim)
    return sims


def assert_same(a, b):
    assert a.n == b.n
    for r in range(a.n):
        assert a.info(r).step == b.info(r).step and a.info(r).stopped == b.info(r).stopped
        for i, bd in enumerate(a.specs[r]["boundaries"]):
            if bd["type"] == "discrete":
                np.testing.assert_array_equal(a.channels(i, r), b.channels(i, r))
        np.testing.assert_array_equal(a.state(r), b.state(r), err_msg=f"realisation {r}")


@pytest.mark.parametrize("shape", SHAPES)
def test_shapes(pkg, synth, shape):
    spec = synth.tiny(shape, serca=min(shape) >= 9)
    a, b = both(pkg, spec, dict(h=6.0, tstop=5.0, seed=3, open_states={"ryr": [0, 1, 2]}), 60, calls=3)
    assert_same(a, b)


def random_model(synth, rng, shape):
    """The reference species on a geometry of random domain blocks, with SERCA pairs across
    random faces (any domains) and channels anywhere."""
    spec = synth.tiny((12, 12, 16))
    coarse = rng.integers(0, 4, size=tuple((n + 2) // 3 for n in shape)).astype(np.uint8)
    vox = np.kron(coarse, np.ones((3, 3, 3), dtype=np.uint8))[:shape[0], :shape[1], :shape[2]]
    spec["voxels"] = np.ascontiguousarray(vox)
    spec["global_size"] = [6.0 * n for n in shape]

    def pairs(n):
        frm = np.stack([rng.integers(0, m, size=n) for m in shape], axis=1)
        to = frm.copy()
        axis = rng.integers(0, 3, size=n)
        step = rng.choice([-1, 1], size=n)
        for i in range(n):
            m = shape[axis[i]]
            to[i, axis[i]] = frm[i, axis[i]] + (step[i] if 0 <= frm[i, axis[i]] + step[i] < m else -step[i])
        return np.concatenate([frm, to], axis=1).astype(np.uint16)

    for bd, n in zip(spec["boundaries"], (7, 4, 300)):
        bd["pairs"] = pairs(n)
    return spec


@pytest.mark.parametrize("shape,react,stoch,dirichlet", [((14, 15, 18), 1, 1, False), ((9, 22, 13), 3, 2, False),
                                                        ((10, 12, 21), 1, 1, True), ((31, 10, 12), 5, 1, False)])
def test_random_geometries(pkg, synth, shape, react, stoch, dirichlet):
    rng = np.random.default_rng(sum(shape))
    spec = random_model(synth, rng, shape)
    if dirichlet:
        spec["fixed_domain_species"] = [(1, 1)]
    dt = 0.95 * 36 / (6 * 220000.0)
    opts = dict(h=6.0, tstop=5.0, seed=4, open_states={"ryr": [0, 2], "p_ryr": [1]}, force_dirichlet=dirichlet,
                dt_update_react=(react + 0.01) * dt, dt_update_stoch=(stoch + 0.01) * dt)
    a, b = both(pkg, spec, opts, 48, calls=2)
    assert_same(a, b)


def test_more_realisations_than_in_flight(pkg, synth):
    """Uneven sizes and models in one batch (the last one has a buffer that binds species 1,
    so the whole batch runs on the general variant), each stopping at its own last step."""
    rng = np.random.default_rng(8)
    dt = 0.95 * 36 / (6 * 220000.0)
    specs = [synth.tiny(s, pryr=k % 2 == 0) for k, s in enumerate([(12, 12, 16), (20, 9, 14), (11, 30, 12)] * 60)]
    opts = [dict(h=6.0, tstop=(20 + k % 7) * dt, seed=17, open_states={"ryr": [k % 7]}) for k in range(len(specs))]
    a, b = both(pkg, specs, opts, 40)
    assert_same(a, b)
    mixed = [random_model(synth, rng, (12, 13, 14)) for _ in range(3)]
    mixed[2]["domain_species"] = {k: dict(v) for k, v in mixed[2]["domain_species"].items()}
    mixed[2]["domain_species"]["cyt"]["buffers"] = [dict(x) for x in mixed[2]["domain_species"]["cyt"]["buffers"]]
    mixed[2]["domain_species"]["cyt"]["buffers"][3]["species"] = [4, 1]
    a, b = both(pkg, mixed, [dict(h=6.0, tstop=5.0, seed=5)] * 3, 30, calls=3)
    assert_same(a, b)


def test_handles_of_different_row_lengths(pkg, synth):
    """A second handle does not change what the first one's launches need."""
    long = pkg.Simulation(synth.tiny((12, 14, 120)), dict(h=6.0, tstop=5.0, seed=1))
    pkg.Simulation(synth.tiny((12, 12, 16)), dict(h=6.0, tstop=5.0, seed=1)).advance(20)
    long.advance(20)
    ref = pkg.Simulation(synth.tiny((12, 14, 120)), dict(h=6.0, tstop=5.0, seed=1))
    ref.set_kernel(1)
    ref.advance(20)
    assert_same(long, ref)
