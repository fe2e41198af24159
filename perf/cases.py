"""Performance cases of the calcium_sparks step: what users of this package have it do.

A case is one call (or the few calls of one output cycle) through the public Python
bindings of libcsparks_cuda.so: time steps of one grid, of an ensemble of equal or of
uneven grids, a whole ensemble job from host memory, the reaction surrogate, the output
path and the surrogate's training gradient.  Models are the seeded synthetic sparks of
synth.py; every realisation starts from a spark in progress (a Gaussian of raised Ca
around the cluster, depleted SR, buffers part of the way to their new equilibrium), so
that no term of the step is trivially zero.

listed()        the cases; draw(rng): one more of the same ranges
prepare()       inputs and handle, as a user's program holds them before the call
run()           one pass
work()          bytes and operations one pass cannot do without
exact()         the same outputs from plain FP64 torch
"""
import importlib
import math

import numpy as np
import torch

PKG = "hpc-ca-phospattern_b200"
SIGMA_MAX = 220000.0          # nm^2/ms, free Ca in the cytosol (synth.species_model)
NS, ND = 5, 5
MLP_IN, MLP_H, MLP_OUT = 8, 64, 5


# ---- the cases ----

def listed():
    return [
        # the smallest calls: a tiny dyad (the grid of the smoke run and of most tests),
        # a few steps per call as an interactive driver or a fine output cadence takes them
        dict(name="grid 12x12x16", kind="grid", nx=12, ny=12, nz=16, steps=64, react=1, stoch=1, tune=0, dirichlet=0),
        # a small dyad as the CLI runs it between two outputs
        dict(name="grid 40x40x36", kind="grid", nx=40, ny=40, nz=36, steps=256, react=1, stoch=1, tune=1, dirichlet=0),
        # the plain single-realisation configuration (0.6 x 0.6 x 0.3 um at 6 nm)
        dict(name="grid 100x100x50", kind="grid", nx=100, ny=100, nz=50, steps=400, react=1, stoch=1, tune=1,
             dirichlet=0),
        # the large single grid (1.2 x 1.2 x 0.6 um at 6 nm, 10x10 RyR lattice)
        dict(name="grid 200x200x100", kind="grid", nx=200, ny=200, nz=100, steps=200, react=1, stoch=1, tune=1,
             dirichlet=0),
        # nothing a multiple of four; reactions every 3 steps, gating every 2, fixed outer
        # faces: the command line's -T, -D and -f
        dict(name="grid 93x75x57 -T3 -D2 -f", kind="grid", nx=93, ny=75, nz=57, steps=300, react=3, stoch=2, tune=0,
             dirichlet=1),
        # many small grids at once, as a parameter sweep over small dyads
        dict(name="ensemble 64 x 36x36x32", kind="ensemble", n=64, nx=36, ny=36, nz=32, steps=200, react=1, tune=0),
        # the batched ensemble of 100x100x50 sparks (clusters of 16-100 RyRs, abort rule
        # 1.5 ms), as many realisations as leave the state well above the L2 cache
        dict(name="ensemble 40 x 100x100x50", kind="ensemble", n=40, nx=100, ny=100, nz=50, steps=300, react=1, tune=1),
        # uneven grids from 64^3 up at 6-10 nm, each with its own dt, reactions every 5 steps
        dict(name="ensemble uneven 8 -T5", kind="uneven", n=8, lo=64, hi=256, steps=150, react=5, tune=1),
        # a whole job from page-locked FP32 host memory: upload, steps, download in one call
        dict(name="job 24 x 100x100x50", kind="job", n=24, nx=100, ny=100, nz=50, steps=200, react=1, tune=0),
        # reactions every 10 steps with the learned surrogate in place of the explicit step
        dict(name="surrogate 24 x 100x100x50", kind="surrogate", n=24, nx=100, ny=100, nz=50, steps=200, react=10,
             tune=0),
        # the output path of one cycle: scalars of every species and domain, a linescan per
        # axis, every field to the host
        dict(name="outputs 200x200x100", kind="outputs", nx=200, ny=200, nz=100),
        # forward and backward of the surrogate's network over a training set
        dict(name="gradient 262144", kind="gradient", pairs=262144),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes over the whole range (log-uniform), odd ones among them."""
    kind = rng.choice(["grid", "grid", "grid", "ensemble", "ensemble", "uneven", "job", "surrogate", "outputs",
                       "gradient"])
    react = rng.choice([1, 1, 1, 2, 3, 5, 10])
    if kind == "grid":
        nx, ny, nz = _log(rng, 12, 220), _log(rng, 12, 220), _log(rng, 16, 110)
        steps = max(16, min(400, int(1.6e9 / (nx * ny * nz))))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=rng.randint(max(16, steps // 2), steps), react=react,
                    stoch=rng.choice([1, 1, 2, 4]), tune=rng.choice([0, 1]), dirichlet=rng.choice([0, 0, 0, 1]))
    if kind in ("ensemble", "job", "surrogate"):
        nx, ny, nz = _log(rng, 24, 130), _log(rng, 24, 130), _log(rng, 24, 64)
        n = _log(rng, 3, max(4, min(64, int((2.0e7 if kind == "ensemble" else 1.2e7) / (nx * ny * nz)))))
        return dict(kind=kind, n=n, nx=nx, ny=ny, nz=nz, steps=rng.randint(80, 200),
                    react=10 if kind == "surrogate" else react, tune=rng.choice([0, 1]) if kind == "ensemble" else 0)
    if kind == "uneven":
        lo = _log(rng, 32, 96)
        return dict(kind=kind, n=rng.randint(3, 8), lo=lo, hi=_log(rng, lo + 16, 200), steps=rng.randint(60, 150),
                    react=rng.choice([1, 5]), tune=rng.choice([0, 1]))
    if kind == "outputs":
        return dict(kind=kind, nx=_log(rng, 24, 200), ny=_log(rng, 24, 200), nz=_log(rng, 20, 100))
    return dict(kind=kind, pairs=_log(rng, 16384, 524288))


# ---- inputs ----

def _mod(name=""):
    return importlib.import_module(PKG + name)


def _uneven_shapes(case):
    rng = np.random.default_rng([case["n"], case["lo"], case["hi"], 5])
    lo, hi = case["lo"], case["hi"]
    return [(int(rng.integers(lo, hi + 1)), int(rng.integers(lo, hi + 1)),
             int(rng.integers(lo, max(lo + 1, hi // 2 + 1)))) for _ in range(case["n"])]


def _models(case, seed):
    """(spec, options) of every realisation of a case: sizes and channel counts from the case,
    positions, phosphorylation and draws from the seed."""
    synth = _mod(".synth")
    rng = np.random.default_rng([seed, 17])
    sizes = np.random.default_rng([case.get(k, 0) for k in ("n", "nx", "ny", "nz", "lo", "hi")])
    kind = case["kind"]
    if kind in ("grid", "outputs"):
        shapes = [(case["nx"], case["ny"], case["nz"])]
        hs = [6.0]
    elif kind == "uneven":
        lo, hi = case["lo"], case["hi"]
        shapes = _uneven_shapes(case)
        hs = [float(sizes.uniform(6.0, 10.0)) for _ in range(case["n"])]
    else:
        shapes = [(case["nx"], case["ny"], case["nz"])] * case["n"]
        hs = [6.0] * case["n"]
    base = {}                                         # geometry without channels, by shape
    out = []
    for r, ((nx, ny, nz), h) in enumerate(zip(shapes, hs)):
        small = min(nx, ny) < 60
        px, py = max(2, int(round(nx * 0.6)) // 2 * 2), max(2, int(round(ny * 0.6)) // 2 * 2)
        patch = ((nx - px) // 2, (ny - py) // 2, px, py)
        nch = int(sizes.integers(4, 26) if small else sizes.integers(16, 101))
        shape_kind = ["compact", "elongated", "fragmented"][int(rng.integers(0, 3))]
        pts = synth.lattice_cluster(rng, nch, (nx, ny, nz), pitch=2 if small else 5, kind=shape_kind, patch=patch)
        # channel 0 of "ryr" is the forced-open trigger, up to half of the others are pRyR
        pmask = np.zeros(len(pts), dtype=bool)
        pmask[1 + rng.permutation(len(pts) - 1)[:int(sizes.uniform(0.0, 0.5) * len(pts))]] = True
        if (nx, ny, nz) not in base:
            base[nx, ny, nz] = synth.spark_model((nx, ny, nz), channels=pts, pryr_mask=pmask, serca=True,
                                                 margin=1 if small else 5, jsr_voxels=3 if small else 5)
        spec = dict(base[nx, ny, nz])
        zj = spec["layout"]["sr_z"][0]

        def pairs(sel, zj=zj, pts=pts):
            c = pts[sel]
            z = np.full(len(c), zj)
            return np.stack([c[:, 0], c[:, 1], z, c[:, 0], c[:, 1], z - 1], axis=1).astype(np.uint16)

        serca = [b for b in spec["boundaries"] if b["name"] == "serca"]
        spec["boundaries"] = [dict(name="ryr", type="discrete", pairs=pairs(~pmask))]
        spec.pop("p_ryr", None)
        if pmask.any():
            spec["boundaries"].append(dict(name="p_ryr", type="discrete", pairs=pairs(pmask)))
            spec["p_ryr"] = dict(synth.P_RYR)
        spec["boundaries"] += serca
        spec["h"] = h
        spec["global_size"] = [k * h for k in (nx, ny, nz)]
        dt = _dt(h)
        # tstop 100 ms: no pass reaches the end of the run
        o = dict(h=h, tstop=100.0, seed=int(rng.integers(1, 1 << 30)), open_states={"ryr": [0]})
        if case.get("react", 1) > 1:
            o["dt_update_react"] = (case["react"] + 0.01) * dt
        if case.get("stoch", 1) > 1:
            o["dt_update_stoch"] = (case["stoch"] + 0.01) * dt
        if case.get("dirichlet"):
            o["force_dirichlet"] = True
        if kind in ("ensemble", "job", "surrogate"):
            o["tabort"] = 1.5
        out.append((spec, o))
    return out


def _dt(h):
    return 0.95 * (1.0 / 6) * h * h / SIGMA_MAX


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _tables(spec, dev, dtype):
    """Per-domain init, k_on, k_off, tot [domain][species] (bound species; 0 where absent)."""
    t = {k: torch.zeros(ND, NS, dtype=torch.float64) for k in ("init", "kon", "koff", "tot")}
    for d, name in enumerate(spec["domains"]):
        ds = spec["domain_species"][name]
        for s in range(NS):
            t["init"][d, s] = ds["init"][s]
        for b in ds["buffers"]:
            s = b["species"][0]
            t["kon"][d, s], t["koff"][d, s], t["tot"][d, s] = b["k_on"], b["k_off"], b["tot"]
    return {k: v.to(dev, dtype) for k, v in t.items()}


def _initial(spec, rng):
    """A spark in progress, FP32 [species][x][y][z] on the device of torch."""
    dev = _device()
    shape = spec["voxels"].shape
    dom = torch.from_numpy(spec["voxels"].astype(np.int64)).to(dev)
    t = _tables(spec, dev, torch.float32)
    amp, dep = float(rng.uniform(2.0, 60.0)), float(rng.uniform(0.05, 0.5))
    width, w = float(rng.uniform(0.06, 0.12)), float(rng.uniform(0.4, 0.9))
    r2 = 0.0
    for a in range(3):
        x = (torch.arange(shape[a], device=dev, dtype=torch.float32) + 0.5) / shape[a] - float(rng.uniform(0.45, 0.55))
        r2 = r2 + (x * x).reshape([-1 if b == a else 1 for b in range(3)])
    g = torch.exp(-r2 / (2 * width * width))
    u = torch.empty((NS,) + shape, device=dev, dtype=torch.float32)
    init = t["init"][dom]
    sr = (dom == 2) | (dom == 3)
    ca = torch.where(sr, init[..., 0] * (1 - dep * g), init[..., 0] + amp * g)
    u[0] = ca
    for s in range(1, NS):
        kon, koff, tot = t["kon"][dom, s], t["koff"][dom, s], t["tot"][dom, s]
        eq = torch.where(tot > 0, tot * ca / (ca + koff / torch.where(kon > 0, kon, torch.ones_like(kon))),
                         torch.zeros_like(tot))
        u[s] = torch.where(tot > 0, init[..., s] + (w if s < 4 else 0.3 * w) * (eq - init[..., s]), init[..., s])
    return u


def _pinned(shape):
    t = torch.empty(shape, dtype=torch.float32, pin_memory=torch.cuda.is_available())
    return t.numpy(), t


def _host_states(models, seed):
    """Page-locked FP32 initial states of every realisation (views of one block) and the
    torch tensors that own the memory."""
    rng = np.random.default_rng([seed, 29])
    views, keep = [], []
    for spec, _ in models:
        a, t = _pinned((NS,) + spec["voxels"].shape)
        t.copy_(_initial(spec, rng))
        views.append(a)
        keep.append(t)
    return views, keep


def _params(seed):
    """Network parameters: the package's initial hidden layers and a small random output
    layer (corrections of a few per cent of their scale, as a trained network gives)."""
    p = _mod().mlp_init(seed % 1000 + 1)
    rng = np.random.default_rng([seed, 43])
    k = MLP_H * MLP_OUT + MLP_OUT
    p[-k:] = (0.02 * rng.standard_normal(k)).astype(np.float32)
    return p


def _pairs(case, seed):
    rng = np.random.default_rng([seed, 57])
    n = case["pairs"]
    x = np.empty((n, MLP_IN), dtype=np.float32)
    x[:, 0] = rng.uniform(-1.0, math.log10(500.0), n) / 3.0
    x[:, 1:6] = rng.random((n, 5))
    x[:, 5] = np.where(rng.random(n) < 0.5, 0.0, x[:, 5])
    x[:, 6] = math.log10(10 * _dt(6.0)) * 0.25
    x[:, 7] = 0.25 * rng.integers(0, 2, n)
    t = np.clip(0.5 * rng.standard_normal((n, MLP_OUT)), -2.0, 2.0).astype(np.float32)
    return x, t


def prepare(case, seed):
    pkg = _mod()
    kind = case["kind"]
    if kind == "gradient":
        x, t = _pairs(case, seed)
        return dict(kind=kind, params=_params(seed), x=x, t=t)
    models = _models(case, seed)
    sim = pkg.Simulation([m[0] for m in models], [m[1] for m in models])
    states, keep = _host_states(models, seed)
    st = dict(kind=kind, sim=sim, states=states, keep=keep, steps=case.get("steps", 0))
    if kind == "surrogate":
        sim.set_surrogate(_params(seed), 1e-4)
    if kind != "job":
        sim.set_states_f32(states)
    if case.get("tune"):
        sim.autotune(repeats=3)
    if kind == "uneven":
        out = [_pinned(u.shape) for u in states]
        st["out"], st["views"] = [a for a, _ in out], [a for a, _ in out]
        st["keep"] = keep + [t for _, t in out]
    elif kind != "outputs":
        a, t = _pinned((len(states),) + states[0].shape)
        st["out"], st["views"] = a, [a[r] for r in range(len(states))]
        st["keep"] = keep + [t]
    if kind == "grid":
        st["discrete"] = [b for b, d in enumerate(models[0][0]["boundaries"]) if d["type"] == "discrete"]
    if kind == "outputs":
        shape = states[0].shape[1:]
        st["offsets"], st["conv"] = [0.5 * n * 6.0 for n in shape], [4.0e4, 4.0e4, 1.6e5]
    return st


def run(st):
    """One pass."""
    kind = st["kind"]
    if kind == "gradient":
        loss, grad = _mod().mlp_gradient(st["params"], st["x"], st["t"])
        return {"grad": grad, "loss": np.float32(loss)}
    sim = st["sim"]
    if kind == "job":
        sim.run_states(st["states"], st["steps"], st["views"])
        return st["out"]
    if kind == "outputs":
        mn, mx, tot, opened = sim.outputs()
        lines = [sim.linescan(1, a, st["offsets"], st["conv"]) for a in range(3)]
        sim.snapshot_async()
        mn, mx, tot = mn[:4], mx[:4], tot[:4]         # these models have no voxel of the fifth domain
        return {"min": mn, "max": mx, "total": tot, "open": opened, "lines": lines, "fields": sim.snapshot_wait()}
    sim.advance(st["steps"])
    sim.states_into_f32(st["views"])
    if kind == "grid":
        return {"state": st["out"], "channels": [sim.channels(b) for b in st["discrete"]]}
    return st["out"]


def work(case):
    """One pass reads the state once and writes it once (the fields may stay on the chip
    between steps); operations: 13 per voxel and diffusing species, 9 per voxel and buffer
    on the steps that take them."""
    kind = case["kind"]
    if kind == "gradient":
        n, w = case["pairs"], MLP_IN * MLP_H + MLP_H * MLP_H + MLP_H * MLP_OUT
        return {"bytes": 4.0 * n * (MLP_IN + MLP_OUT), "flops": 6.0 * n * w}
    if kind == "uneven":
        vox = float(sum(a * b * c for a, b, c in _uneven_shapes(case)))
    else:
        vox = float(case.get("n", 1)) * case["nx"] * case["ny"] * case["nz"]
    if kind == "outputs":
        return {"bytes": vox * (4 * NS + 8 * NS + 1), "flops": vox * NS * 4}
    steps = case["steps"]
    diffusing = 1 + 1 / 11 + 1 / 9 + 1                 # Ca, Fluo, CMDN, ATP and their substeps
    return {"bytes": vox * (8 * NS + 1.0), "flops": vox * steps * (13 * diffusing + 9 * 4 / case["react"])}


# ---- exact: the same step in FP64 torch ----

def _substeps(spec, h, dt):
    """Global diffusive species and their substeps (0.95 h^2 / 6 sigma_s over dt, floored)."""
    smax = [0.0] * NS
    for ds in spec["domain_species"].values():
        for s, v in zip(ds["diffusive"], ds["sigma"]):
            smax[s] = max(smax[s], v)
    top = max(smax)
    sub = {}
    for s in range(NS):
        if smax[s] > 0:
            sdt = dt if abs(top - smax[s]) < 1e-12 else 0.95 * (1.0 / 6) * h * h / smax[s]
            sub[s] = max(1, int(math.floor(sdt / dt)))
    return sub


def _uniforms(seed, stream, boundary, nch, first, last):
    """Philox4x32-10 uniforms [step][channel] of the time indices first..last (53 bits of the
    first two words; counter = channel, boundary, step; key = seed, stream)."""
    m32 = np.uint64(0xFFFFFFFF)
    ch, ti = np.meshgrid(np.arange(nch, dtype=np.uint64), np.arange(first, last + 1, dtype=np.uint64))
    c = [ch, np.full_like(ch, boundary), ti, np.zeros_like(ch)]
    k0, k1 = seed & 0xFFFFFFFF, (stream ^ (seed >> 32)) & 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1),
             p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    hi, lo = (c[0] >> np.uint64(5)).astype(np.float64), (c[1] >> np.uint64(6)).astype(np.float64)
    return (hi * 67108864.0 + lo) / 2.0**53


def _serca(dt, h, u0, u1, density):
    """SERCA flux of a pair (cytosol u0, SR u1): the three-state cycle."""
    ti2, ts2 = (u0 / 1000 / 0.9) ** 2, (u1 / 1000 / 2.24) ** 2
    H, ATP, ADP = 1e-4, 5.0, 36.3e-3
    t1, thi, ths, th = H / 1.09e-5, H * H / 3.54e-3, H * H / 1.05e-8, H / 7.24e-5
    di = ti2 + ti2 * thi + thi * (1 + t1)
    ds = ts2 * th + th + ths * (1 + th)
    p1, p2, p3 = 25900 * ATP, 2540 * ti2 / di, 20.5 * ths / ds
    m1, m2, m3 = 16 * thi / di, 67200 * ADP * ts2 * th / ds, 149.0
    s = (p2 * p3 + m1 * p3 + m1 * m2) + (p1 * p3 + m2 * p1 + m2 * m3) + (p1 * p2 + m3 * m1 + m3 * p2)
    v = (p1 * p2 * p3 - m1 * m2 * m3) / s
    return dt * (h * h * density * v * (1e-3 / 6e17)) / (1e-24 * h**3)


class _Fp64Step:
    """The step of one realisation in FP64."""

    def __init__(self, spec, opts, stream, case, u0):
        dev = _device()
        f64 = torch.float64
        self.dev, self.case = dev, case
        self.h = h = spec["h"]
        self.dt = dt = _dt(h)
        self.react, self.stoch = case.get("react", 1), case.get("stoch", 1)
        self.u = u0.to(dev, f64)
        dom = torch.from_numpy(spec["voxels"].astype(np.int64)).to(dev)
        self.dom, self.t = dom, _tables(spec, dev, f64)
        self.kon, self.koff, self.tot = (self.t[k][dom].permute(3, 0, 1, 2).contiguous() for k in ("kon", "koff", "tot"))
        self.sub = _substeps(spec, h, dt)
        conn = torch.from_numpy(np.asarray(spec["domain_connections"], dtype=np.float64))
        self.coef = {}
        for s, n in self.sub.items():
            sig = [dict(zip(spec["domain_species"][d]["diffusive"], spec["domain_species"][d]["sigma"])).get(s, 0.0)
                   for d in spec["domains"]]
            c = torch.zeros(ND, ND, dtype=f64)
            for a in range(ND):
                for b in range(ND):
                    if sig[a] and sig[b] and conn[a, b]:
                        c[a, b] = dt * 0.5 * (sig[a] + sig[b]) / (h * h) * n
            c = c.to(dev)
            self.coef[s] = [c[dom.narrow(ax, 0, dom.shape[ax] - 1), dom.narrow(ax, 1, dom.shape[ax] - 1)]
                            for ax in range(3)]
        sh = spec["voxels"].shape

        def lin(v):
            v = v.astype(np.int64)
            return torch.from_numpy((v[:, 0] * sh[1] + v[:, 1]) * sh[2] + v[:, 2]).to(dev)

        self.pairs = []
        for b, bd in enumerate(spec["boundaries"]):
            v0, v1 = lin(bd["pairs"][:, :3]), lin(bd["pairs"][:, 3:])
            if bd["type"] == "discrete":
                n = len(bd["pairs"])
                state = torch.zeros(n, dtype=torch.bool, device=dev)
                law = spec["ryr"] if bd["name"] == "ryr" else spec["p_ryr"]
                if bd["name"] in opts["open_states"]:
                    state[opts["open_states"][bd["name"]]] = True
                else:
                    # the initial draw of the p_ryr channels reads the ryr boundary's Ca (resting everywhere)
                    ko, kc = self._rates(law, torch.full((n,), 0.14, dtype=f64, device=dev))
                    first = torch.from_numpy(_uniforms(opts["seed"], stream, b, n, 0, 0)[0]).to(dev)
                    state = first > kc / (ko + kc)
                uni = torch.from_numpy(_uniforms(opts["seed"], stream, b, n, 1, case["steps"])).to(dev)
                k0 = math.exp(-2 * dt * 1e15 / (2 * 96485.0) * law["i_unitary"] / (1300.0 - 0.1) / h**3)
                self.pairs.append(dict(v0=v0, v1=v1, state=state, law=law, uni=uni, k0=k0))
            else:
                self.pairs.append(dict(v0=v0, v1=v1, density=spec["serca"]["density"]))
        self.dinit = None
        if case.get("dirichlet"):
            self.dinit = self.t["init"][dom, 0]
            self.face = torch.ones_like(dom, dtype=torch.bool)
            self.face[1:-1, 1:-1, 1:-1] = False
        self.net = None

    @staticmethod
    def _rates(law, c):
        ko = torch.clamp((c / law["Kd_open"]) ** law["n_open"], law["k_min_open"], law["k_max_open"])
        kc = torch.clamp((c / law["Kd_close"]) ** law["n_close"], law["k_min_close"], law["k_max_close"])
        return ko, kc

    def channels(self):
        return [p["state"].to(torch.int32).cpu().numpy() for p in self.pairs if "state" in p]

    def step(self, ti):
        u, new = self.u, self.u.clone()
        for s, n in self.sub.items():
            if ti % n:
                continue
            for ax in range(3):
                m = u.shape[1 + ax]
                j = self.coef[s][ax] * (u[s].narrow(ax, 1, m - 1) - u[s].narrow(ax, 0, m - 1))
                new[s].narrow(ax, 0, m - 1).add_(j)
                new[s].narrow(ax, 1, m - 1).sub_(j)
        ca, flat = u[0].reshape(-1), new[0].reshape(-1)
        for p in self.pairs:
            a, b = ca[p["v0"]], ca[p["v1"]]
            if "state" in p:
                if ti % self.stoch == 0:
                    ko, kc = self._rates(p["law"], b)
                    dts, r = self.dt * self.stoch, p["uni"][ti - 1]
                    p["state"] = torch.where(p["state"], ~(r <= dts * kc), r <= dts * ko)
                j = torch.where(p["state"], (a - b) * (1 - p["k0"]) / 2, torch.zeros_like(a))
            else:
                j = _serca(self.dt, self.h, a, b, p["density"])
            flat.index_add_(0, p["v1"], j)
            flat.index_add_(0, p["v0"], -j)
        if ti % self.react == 0:
            db, dc = self._reaction()
            for s in range(1, NS):
                new[s] += db[s - 1]
            new[0] += dc
        if self.dinit is not None:
            new[0] = torch.where(self.face, self.dinit, new[0])
        self.u = new

    def _rhs(self, c, b):
        return [self.kon[s] * (self.tot[s] - b[s - 1]) * c - self.koff[s] * b[s - 1] for s in range(1, NS)]

    def _reaction(self):
        dtr = self.dt * self.react
        c, b = self.u[0], [self.u[s] for s in range(1, NS)]
        g = self._rhs(c, b)
        db = [dtr * x for x in g]
        dc = -sum(db)
        if self.net is None:
            return db, dc
        # plain integrator: the same update `react` times at dt
        cc, bb = c, b
        for _ in range(self.react):
            gg = self._rhs(cc, bb)
            bb = [x + self.dt * y for x, y in zip(bb, gg)]
            cc = cc - self.dt * sum(gg)
        pdb, pdc = [x - y for x, y in zip(bb, b)], cc - c
        # network: correction of the explicit step, scaled by the second-order term
        kon, koff, tot = (self.t[k] for k in ("kon", "koff", "tot"))
        on = tot > 0
        stiff = (kon * tot).sum(1) + torch.where(on, koff + 500.0 * kon, torch.zeros_like(koff)).max(1).values
        eligible = (on.any(1) & (dtr * stiff <= 0.25))[self.dom]
        some = on.any(1)[self.dom]
        G = sum(g).abs()
        one = torch.ones_like(c)
        S, safe = [], [torch.where(self.tot[s] > 0, self.tot[s], one) for s in range(1, NS)]
        for s in range(1, NS):
            lam = self.koff[s] + self.kon[s] * c
            S.append(0.5 * dtr * dtr * (lam * g[s - 1].abs() + self.kon[s] * (self.tot[s] - b[s - 1]) * G) / safe[s - 1])
        away = torch.stack(S).max(0).values > 1e-8
        idx = (eligible & away).reshape(-1).nonzero().reshape(-1)
        x = torch.zeros(idx.numel(), MLP_IN, dtype=torch.float64, device=self.dev)
        x[:, 0] = torch.log10(torch.clamp(c.reshape(-1)[idx], min=1e-3)) / 3
        for s in range(1, NS):
            x[:, s] = (b[s - 1] / safe[s - 1] * (self.tot[s] > 0)).reshape(-1)[idx]
        x[:, 6], x[:, 7] = math.log10(dtr) * 0.25, 0.25 * self.dom.reshape(-1)[idx].double()
        w1, b1, w2, b2, w3, b3 = self.net
        t = torch.relu(torch.relu(x @ w1 + b1) @ w2 + b2) @ w3 + b3
        at = [v.reshape(-1)[idx] for v in (c, *b)]
        ks = [[k[s].reshape(-1)[idx] for s in range(1, NS)] for k in (self.kon, self.koff, self.tot)]
        ndb = [dtr * g[s - 1].reshape(-1)[idx] + ks[2][s - 1] * S[s - 1].reshape(-1)[idx] * t[:, s - 1]
               for s in range(1, NS)]
        ndc = -sum(ndb)
        worst = torch.zeros_like(ndc)
        for s in range(1, NS):
            g1 = ks[0][s - 1] * (ks[2][s - 1] - at[s] - ndb[s - 1]) * (at[0] + ndc) - ks[1][s - 1] * (at[s] + ndb[s - 1])
            r = (ndb[s - 1] - 0.5 * dtr * (g[s - 1].reshape(-1)[idx] + g1)).abs() / safe[s - 1].reshape(-1)[idx]
            worst = torch.maximum(worst, r)
        ok = worst <= 1e-4
        plain = some & ~eligible
        out = []
        for s, (e, p) in enumerate(zip([*db, dc], [*pdb, pdc])):
            v = torch.where(plain, p, e)
            v.reshape(-1)[idx] = torch.where(ok, ndb[s] if s < NS - 1 else ndc, p.reshape(-1)[idx])
            out.append(v)
        return out[:-1], out[-1]


def _unpack(p):
    shapes, out, o = ((MLP_IN, MLP_H), (MLP_H,), (MLP_H, MLP_H), (MLP_H,), (MLP_H, MLP_OUT), (MLP_OUT,)), [], 0
    for s in shapes:
        n = int(np.prod(s))
        out.append(torch.from_numpy(np.asarray(p[o:o + n], dtype=np.float64)).reshape(s).to(_device()))
        o += n
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        x, t = (torch.from_numpy(a).to(_device(), torch.float64) for a in _pairs(case, seed))
        w = [v.requires_grad_() for v in _unpack(_params(seed))]
        y = torch.relu(torch.relu(x @ w[0] + w[1]) @ w[2] + w[3]) @ w[4] + w[5]
        loss = ((y - t) ** 2).mean()
        loss.backward()
        return {"grad": torch.cat([v.grad.reshape(-1) for v in w]).cpu().numpy(), "loss": np.float64(loss.item())}
    models = _models(case, seed)
    states, _ = _host_states(models, seed)
    if kind == "outputs":
        return _exact_outputs(models[0][0], states[0])
    results, channels = [], None
    for r, ((spec, opts), u0) in enumerate(zip(models, states)):
        sim = _Fp64Step(spec, opts, r, case, torch.from_numpy(u0))
        if kind == "surrogate":
            sim.net = _unpack(_params(seed))
        for ti in range(1, case["steps"] + 1):
            sim.step(ti)
        results.append(sim.u.cpu().numpy())
        channels = sim.channels()
    if kind == "uneven":
        return results
    out = np.stack(results)
    return {"state": out, "channels": channels} if kind == "grid" else out


def _exact_outputs(spec, u0):
    dom = torch.from_numpy(spec["voxels"].astype(np.int64)).to(_device())
    u = torch.from_numpy(u0).to(_device(), torch.float64)
    h = spec["h"]
    f32 = np.finfo(np.float32)
    mn, mx, tot = (np.zeros((4, NS)) for _ in range(3))
    for d in range(4):
        m = dom == d
        for s in range(NS):
            v = u[s][m]
            # the reductions start from FLT_MAX and FLT_MIN
            mn[d, s] = min(float(f32.max), v.min().item()) if v.numel() else float(f32.max)
            mx[d, s] = max(float(f32.tiny), v.max().item()) if v.numel() else float(f32.tiny)
            tot[d, s] = v.sum().item() * h**3
    offsets, conv = [0.5 * n * 6.0 for n in dom.shape], [4.0e4, 4.0e4, 1.6e5]

    def gauss(x, s):
        return np.exp(-x * x / 2 / s) / math.sqrt(2 * math.pi * s)

    lines = []
    for a in range(3):
        f = u[1]
        for b in (2, 1, 0):
            if b != a:
                w = torch.from_numpy(gauss(offsets[b] - np.arange(dom.shape[b]) * h, conv[b])).to(f)
                f = (f * w.reshape([-1 if q == b else 1 for q in range(3)])).sum(b, keepdim=True)
        f = f.reshape(-1).cpu().numpy()
        i = np.arange(len(f))
        lines.append(gauss((i[:, None] - i[None, :]) * h, conv[a]) @ f)
    return {"min": mn, "max": mx, "total": tot, "open": None, "lines": lines, "fields": u.cpu().numpy()}
