"""The step kernel on models that are not of the reference model's shape -- fixed values and
Dirichlet faces, a second fixed-point species, fewer and more species, a species that diffuses
faster than Ca, buffers that bind another species than Ca -- alone and in batches with the
reference model, which then runs on the same variant: fields and channel states bitwise those
of the direct kernel, with the surrogate where it is supported.  And none of them is slower
than it was with one launch per step: bounds in terms of the reference model's step."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = 0.95 * 36 / (6 * 220000.0)


def copied(spec):
    spec["species"] = list(spec["species"])
    spec["domain_species"] = {d: dict(v, diffusive=list(v["diffusive"]), sigma=list(v["sigma"]), init=list(v["init"]),
                                      buffers=[dict(b) for b in v["buffers"]])
                              for d, v in spec["domain_species"].items()}
    return spec


def species(n, diffusing=False):
    """n species: those beyond TRPN are Ca buffers of the cytosol and the cleft."""
    def change(spec):
        copied(spec)
        spec["species"] = spec["species"][:n] + ["X%d" % k for k in range(5, n)]
        for d, ds in spec["domain_species"].items():
            ds["buffers"] = [b for b in ds["buffers"] if b["species"][0] < n]
            keep = [i for i, s in enumerate(ds["diffusive"]) if s < n]
            ds["diffusive"], ds["sigma"] = [ds["diffusive"][i] for i in keep], [ds["sigma"][i] for i in keep]
            ds["init"] = ds["init"][:n]
            for k in range(5, n):
                ca, kon, koff, tot = ds["init"][0], 0.05 / (k - 3), 0.1, 30.0 + k
                if d in ("jsr", "nsr", "tt"):
                    ds["init"].append(0.0)
                    continue
                ds["buffers"].append(dict(species=[k, 0], k_on=kon, k_off=koff, tot=tot))
                ds["init"].append(tot * ca / (ca + koff / kon))
                if diffusing:
                    ds["diffusive"].append(k)
                    ds["sigma"].append(20000.0)
        return spec
    return change


def trpn_diffuses(spec):
    copied(spec)
    for d in ("cyt", "cleft"):
        spec["domain_species"][d]["diffusive"].append(4)
        spec["domain_species"][d]["sigma"].append(20000.0)
    return spec


def two_fixed_point(spec):
    copied(spec)
    for d in ("cyt", "cleft"):
        ds = spec["domain_species"][d]
        ds["diffusive"], ds["sigma"] = [0, 1, 2], ds["sigma"][:3]
    return spec


def fast_atp(spec):
    """Ca (and its SERCA flux) every second step only."""
    copied(spec)
    for d in ("cyt", "cleft"):
        spec["domain_species"][d]["sigma"] = spec["domain_species"][d]["sigma"][:3] + [500000.0]
    return spec


def binds_fluo(spec):
    copied(spec)["domain_species"]["cyt"]["buffers"][3]["species"] = [4, 1]
    return spec


def fixed_value(spec):
    return dict(spec, fixed_domain_species=[(1, 1), (0, 4)])


def same(spec):
    return spec


MODELS = {"reference": (same, {}), "dirichlet": (same, dict(force_dirichlet=True)), "fixed value": (fixed_value, {}),
          "two fixed point": (two_fixed_point, {}), "3 species": (species(3), {}), "1 species": (species(1), {}),
          "TRPN diffuses": (trpn_diffuses, {}), "fast ATP": (fast_atp, {}), "binds Fluo": (binds_fluo, {}),
          "6 species": (species(6), {}), "8 species": (species(8), {}), "8 diffusing": (species(8, True), {})}
SURROGATE = ["reference", "dirichlet", "fixed value", "two fixed point", "3 species", "TRPN diffuses", "6 species"]


def build(synth, names, shape, **more):
    specs, opts = [], []
    for k, name in enumerate(names):
        change, o = MODELS[name]
        specs.append(change(synth.tiny(shape)))
        opts.append(dict(dict(h=6.0, tstop=5.0, seed=3 + k, open_states={"ryr": [0, 1, 2]}), **o, **more))
    return specs, opts


def check_same(pkg, specs, opts, steps, surrogate=False):
    sims = []
    for kernel in (0, 1):
        sim = pkg.Simulation(specs, opts)
        sim.set_kernel(kernel)
        if surrogate:
            p = pkg.mlp_init(5)
            rng = np.random.default_rng(43)
            p[-325:] = (0.02 * rng.standard_normal(325)).astype(np.float32)
            sim.set_surrogate(p, 1e-4)
        sim.advance(steps)
        sims.append(sim)
    a, b = sims
    for r in range(a.n):
        for i, bd in enumerate(specs[r]["boundaries"]):
            if bd["type"] == "discrete":
                np.testing.assert_array_equal(a.channels(i, r), b.channels(i, r))
        u, v = a.state(r), b.state(r)
        assert np.isfinite(u).all()
        np.testing.assert_array_equal(u, v, err_msg=f"realisation {r}")
    a.close()
    b.close()


@pytest.mark.parametrize("shape", [(12, 12, 16), (13, 21, 18)])
@pytest.mark.parametrize("name", list(MODELS))
def test_alone(pkg, synth, name, shape):
    for react in (1, 3):
        specs, opts = build(synth, [name], shape, dt_update_react=(react + 0.01) * DT)
        check_same(pkg, specs, opts, 30)


@pytest.mark.parametrize("name", [m for m in MODELS if m != "reference"])
def test_in_a_batch_with_the_reference_model(pkg, synth, name):
    specs, opts = build(synth, ["reference", name, "reference"], (13, 12, 18))
    check_same(pkg, specs, opts, 24)


@pytest.mark.parametrize("name", SURROGATE)
def test_surrogate_in_a_batch(pkg, synth, name):
    specs, opts = build(synth, ["reference", name], (13, 12, 18), dt_update_react=(3 if name != "fast ATP" else 4) * DT * 1.001)
    check_same(pkg, specs, opts, 24, surrogate=True)


def step_us(pkg, synth, change, o, n=24, steps=60):
    specs = [change(synth.spark_model((100, 100, 50))) for _ in range(n)]
    opts = [dict(dict(h=6.0, tstop=50.0, seed=k, open_states={"ryr": [0]}), **o) for k in range(n)]
    sim = pkg.Simulation(specs, opts)
    sim.advance(steps)
    best = 1e9
    for _ in range(4):
        t = time.perf_counter()
        sim.advance(steps)
        best = min(best, time.perf_counter() - t)
    sim.close()
    return best / steps * 1e6


@pytest.mark.parametrize("name,bound", [("dirichlet", 2.0), ("two fixed point", 2.0), ("binds Fluo", 4.1), ("3 species", 1.55),
                                        ("8 species", 6.8)])
def test_ensemble_not_slower_than_launch_per_step(pkg, synth, name, bound):
    """24 grids of 100x100x50: with a launch per step these models took 213, 209, 428, 165 and
    713 us per step; the reference model's step takes 104 us now."""
    ref = step_us(pkg, synth, *MODELS["reference"])
    us = step_us(pkg, synth, *MODELS[name])
    assert us < bound * ref, (us, ref)
