"""The work that users have the framework do, as cases that a timing program can run.

Kinds of cases, by the public call that each goes through:

  rhs1d   Engine.rhs             one right-hand side on host arrays, as a GSL caller registers it
  step1d  Engine.evolve_apply    one accepted RKF45 step on a host array, the reference's own loop body
  run1d   Engine.set_states / run / get_states
                                 a forecast cycle of one member or of a ragged ensemble: states in,
                                 one window of output samples on the device, states out
  rhs2d   Engine2D.rhs           one 2D right-hand side on host arrays
  run2d   Engine2D.set_state / run_to_time / state_into
                                 the same cycle in 2D
  train   learned.MLP.set_params / train / params
                                 training rounds of the learned depth operator's network

Everything but the network is FP64, which is the only precision the solver has; the network is FP32.
Grids are powers of two because the device engine takes no others; what is ragged is the members of
an ensemble, the 2D sides, the windows and the number of training records.
"""
import functools
import json
import math
import os
import tempfile

import numpy as np
import torch

import hawassi_c_b200 as hw
from hawassi_c_b200 import decks, decks2d, learned
from hawassi_c_b200.engine2d import Engine2D

G = 9.80665
TOL = dict(eps_abs=1e-8, eps_rel=1e-6)   # the tolerances of every configuration of the benchmark
DT = 0.05                                # output interval of the 1D decks (s)
T_END = 102.36                           # 2048 influx samples
RHS_PER_RAD = 100.0                     # RHS evaluations per second of time and unit of the grid's edge frequency


def listed():
    return [
        # a GSL program's RHS callback on the smallest grid in use: launch and copy latency
        dict(name="rhs 1D 512 flat", kind="rhs1d", nx=512, model="HS2"),
        # the reference's loop body, gsl_odeiv_evolve_apply, on a barred beach with breaking (three
        # reference depths), one host round trip a step
        dict(name="step 1D 4096 bar breaking", kind="step1d", nx=4096, model="HS2", bottom="bar", nref=3,
             breaking=True),
        # one wave tank: 200 m, flat, three gauges, in the slice that its benchmark uses
        dict(name="run 1D 4096 flat gauges", kind="run1d", nx=4096, nx_max=4096, members=1, model="HS2", bottom="flat",
             nref=3, breaking=False, gauges=3, slice=512, window=10),
        # the largest single 1D run: 1:30 slope, third order, 16 reference depths, breaking
        dict(name="run 1D 16384 slope HS3", kind="run1d", nx=16384, nx_max=16384, members=1, model="HS3",
             bottom="slope", nref=16, breaking=True, gauges=0, slice=0, window=1),
        # the throughput workload: a ragged ensemble of flat tanks with breaking
        dict(name="run 1D ensemble 256 ragged", kind="run1d", nx=2048, nx_max=16384, members=256, model="HS2",
             bottom="flat", nref=3, breaking=True, gauges=0, slice=0, window=3),
        # random bathymetries under the plain 16-reference operator: what the learned operator's
        # training records and its fallback come from
        dict(name="run 1D 17 bathymetries K16", kind="run1d", nx=4096, nx_max=16384, members=17, model="HS2",
             bottom="bumps", nref=16, breaking=False, gauges=0, slice=0, window=2),
        # the smallest 2D call
        dict(name="rhs 2D 64x64 flat", kind="rhs2d", nx=64, ny=64),
        # an ordinary 2D basin with a flat bottom
        dict(name="run 2D 256x128 flat", kind="run2d", nx=256, ny=128, model=2, bottom="flat", nref=2, breaking=False,
             window=0.4),
        # the same basin in third order
        dict(name="run 2D 512x256 flat HS3", kind="run2d", nx=512, ny=256, model=3, bottom="flat", nref=2,
             breaking=False, window=0.2),
        # the largest 2D run: harbour wall, shoal, breaking (whose update symmetrises part of the RHS, as the
        # reference's does, and so asks for some twenty times the steps of a run without it)
        dict(name="run 2D 1024x1024 harbour", kind="run2d", nx=1024, ny=1024, model=2, bottom="harbour", nref=2,
             breaking=True, window=0.01),
        # the learned operator's form in 2D: four reference depths
        dict(name="run 2D 512x512 shoal K4", kind="run2d", nx=512, ny=512, model=2, bottom="shoal", nref=4,
             breaking=False, window=0.1),
        # training rounds on the records of four bathymetries
        dict(name="train 65536 records", kind="train", records=65536, batch=4096, epochs=3),
    ]


def draw(rng):
    def pow2(lo, hi):
        return 1 << rng.randint(lo, hi)

    kind = rng.choice(["rhs1d", "step1d", "single", "single", "ensemble", "ensemble", "rhs2d", "run2d", "run2d",
                       "run2d", "train"])
    if kind == "rhs1d":
        return dict(kind=kind, nx=pow2(8, 14), model=rng.choice(["HS1", "HS2", "HS2"]))
    if kind == "step1d":
        bottom = rng.choice(["flat", "bar", "slope"])
        return dict(kind=kind, nx=pow2(9, 13), model=rng.choice(["HS2", "HS2", "HS3"]), bottom=bottom,
                    nref=rng.choice([2, 3]), breaking=rng.random() < 0.5)
    if kind == "single":
        bottom = rng.choice(["flat", "bar", "slope", "bumps"])
        nx = pow2(9, 14)
        return dict(kind="run1d", nx=nx, nx_max=nx, members=1, model=rng.choice(["HS1", "HS2", "HS2", "HS3"]),
                    bottom=bottom, nref=rng.choice([2, 3, 4, 16]), breaking=rng.random() < 0.5,
                    gauges=rng.randint(0, 5), slice=512 if nx <= 8192 and rng.random() < 0.5 else 0,
                    window=rng.randint(1, 3 if bottom != "flat" and nx > 4096 else 10))
    if kind == "ensemble":
        bottom = rng.choice(["flat", "flat", "bumps"])
        members = int(round(2 ** rng.uniform(1, 7))) if bottom == "flat" else int(round(2 ** rng.uniform(1, 4)))
        lo = rng.randint(9, 12)
        return dict(kind="run1d", nx=1 << lo, nx_max=pow2(lo, 14), members=members, model="HS2", bottom=bottom,
                    nref=rng.choice([3, 4, 16]), breaking=bottom == "flat" and rng.random() < 0.7, gauges=0, slice=0,
                    window=rng.randint(1, 4 if bottom == "flat" else 2))
    if kind == "rhs2d":
        return dict(kind=kind, nx=pow2(6, 9), ny=pow2(6, 9))
    if kind == "run2d":
        nx = pow2(6, 10)
        ny = 1 << rng.randint(6, min(10, 18 - int(math.log2(nx))))
        bottom = rng.choice(["flat", "flat", "shoal", "shoal"])
        nref = rng.choice([2, 2, 3, 4, 8]) if bottom == "shoal" else 2
        model = rng.choice([1, 2, 2, 3])
        breaking = model == 2 and nref == 2 and rng.random() < 0.5
        return dict(kind=kind, nx=nx, ny=ny, model=model, bottom=bottom, nref=nref, breaking=breaking,
                    window=rng.choice([0.005, 0.01, 0.015] if breaking else [0.1, 0.15, 0.2]))
    batch = rng.choice([512, 1000, 2048, 4096])
    return dict(kind="train", records=int(2 ** rng.uniform(12, 16)) | 1, batch=batch, epochs=rng.randint(1, 3))


# ---------------------------------------------------------------------------
# 1D decks and sea states
# ---------------------------------------------------------------------------
_ROOT = tempfile.mkdtemp(prefix="hw_cases_")


def _frac(m, c):
    return (0.5 + m * c) % 1.0


def _member(case, m):
    """Parameters of member m: the ensemble's ranges (depth 0.5-2 m, Tp 1.5-3 s, gamma 1-5), the wave
    height by a significant steepness of 0.01 to 0.022: crests above the breaking threshold are tested on
    every RHS, few break (a run of breaking crests is chaotic and says nothing about rounding)."""
    levels = int(math.log2(case["nx_max"] // case["nx"])) + 1
    nx = case["nx"] << ((m * 7 + m // 4) % levels)
    bottom = case["bottom"]
    length = nx * (0.05 if bottom in ("flat", "bar") else 400.0 / 16384)
    Tp = 1.5 + 1.5 * _frac(m, 0.754877666)
    depth = 0.5 + 1.5 * _frac(m, 0.618033989) if bottom == "flat" else (2.0 if bottom == "bumps" else 1.0)
    lam = 2 * math.pi / decks2d.invers_omega(2 * math.pi / Tp, depth)
    Hs = min((0.01 + 0.012 * _frac(m, 0.569840291)) * lam, 0.2 * depth)
    bath = None
    if bottom == "bar":
        x = np.linspace(0.0, length, nx)
        bath = 1.0 - 0.6 * np.exp(-((x - 0.55 * length) / (0.1 * length)) ** 4)
    elif bottom == "slope":
        bath = decks.slope_bathymetry(nx, length, h0=1.0, x_toe=0.375 * length, slope=0.95 / (0.075 * 400 / 16384 * nx + 20),
                                      h_min=0.05 if nx >= 8192 else 0.3)
    elif bottom == "bumps":
        bath = decks.bump_bathymetry(nx, length, m, h_min=0.05 if nx >= 8192 else 0.3, h_max=2.0)
        depth = float(bath.max())
    return dict(nx=nx, length=length, depth=depth, bath=bath, Hs=Hs, Tp=Tp, gamma=1.0 + 4.0 * _frac(m, 0.438579021))


@functools.lru_cache(maxsize=None)
def _decks(key):
    """The deck directories of a case (written once: a user's decks lie on disk)."""
    case = json.loads(key)
    paths = []
    base = tempfile.mkdtemp(dir=_ROOT)
    for m in range(case["members"]):
        p = _member(case, m)
        L = p["length"]
        gauges = [L * (0.3 + 0.5 * g / max(case["gauges"], 1)) for g in range(case["gauges"])]
        paths.append(decks.write_deck(
            os.path.join(base, str(m)), nx=p["nx"], length=L, depth=p["depth"], bath=p["bath"], model=case["model"],
            breaking=case["breaking"], T_end=T_END, dt=DT, Hs=p["Hs"], Tp=p["Tp"], gamma=p["gamma"],
            damp=(0.05 * L, 0.05 * L), wavename=case["wavename"], gauges=gauges))
    return paths


def _full(case):
    """A 1D case with every option that its kind leaves out."""
    return {**dict(nx_max=case["nx"], members=1, bottom="flat", nref=3, breaking=False, gauges=0, slice=0, window=1,
                   wavename="zero" if case["kind"] == "rhs1d" else "jonswap"), **case, "name": ""}


def _jonswap(w, Hs, Tp, gamma):
    wp = 2 * math.pi / Tp
    w = np.maximum(w, 1e-3 * wp)
    sig = np.where(w <= wp, 0.07, 0.09)
    return w ** -5.0 * np.exp(-1.25 * (wp / w) ** 4) * gamma ** np.exp(-((w - wp) ** 2) / (2 * (sig * wp) ** 2))


def _sea(p, rng):
    """A sea state that fills the tank: a seeded JONSWAP sum running right, let down over shallow water
    and to rest in the damping zones, within the third-order alias band; the reference's spectral layout."""
    nx, L, h = p["nx"], p["length"], p["depth"]
    k = 2 * math.pi * np.fft.rfftfreq(nx, d=L / (nx - 1))
    k[0] = k[1]
    w = np.sqrt(G * k * np.tanh(k * h))
    cg = 0.5 * w / k * (1 + 2 * k * h / np.sinh(np.minimum(2 * k * h, 500.0)))
    amp = np.sqrt(_jonswap(w, p["Hs"], p["Tp"], p["gamma"]) * cg)
    amp[0] = 0.0
    amp[nx // 6 - 2:] = 0.0
    eh = amp * np.exp(2j * math.pi * rng.random(k.size))
    eta, u = np.fft.irfft(eh, nx), np.fft.irfft(eh * (G * k / w), nx)
    taper = np.minimum(1.0, np.minimum(np.arange(nx), nx - 1 - np.arange(nx)) / (0.1 * nx))
    shape = np.sin(0.5 * math.pi * taper) ** 2 * p["Hs"] / (4 * eta.std())
    if p["bath"] is not None:
        shape = shape * np.minimum(1.0, p["bath"] / (6.0 * p["Hs"]))
    out = []
    for f in (eta * shape, u * shape):
        s = np.fft.rfft(f)
        s[nx // 6 - 2:] = 0.0
        s = np.fft.fft(np.fft.irfft(s, nx))
        s[nx // 6 - 2:nx - (nx // 6 - 2) + 1] = 0.0
        out += [s.real, s.imag]
    return np.concatenate(out)


def _seas(case, seed):
    rng = np.random.default_rng([seed, 11])
    return [_sea(_member(case, m), rng) for m in range(case["members"])]


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    v = t.numpy()
    v[:] = a.ravel()
    return v


# ---------------------------------------------------------------------------
# 2D tables and sea states
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _tables(key):
    """The set-up tables of a 2D run (built once: a user keeps them beside the engine)."""
    c = json.loads(key)
    nx, ny = c["nx"], c["ny"]
    kw = dict(nx=nx, ny=ny, n_freq=48, n_dir=16, t_end=30.0, dt=0.1, model=c["model"], seed=1)
    if c["bottom"] == "harbour":
        return decks2d.config5(**kw)
    Lx, Ly = 0.6 * nx, 0.6 * ny
    kw.update(Lx=Lx, Ly=Ly, depth=3.0, Hs=0.3, Tp=4.0, damp=0.1 * min(Lx, Ly), x_line=0.15 * Lx, nadj=0.5,
              breaking=c["breaking"])
    if c["bottom"] == "shoal":
        tb = decks2d.tables(bathymetry="shoal", shallow=0.6, ninterp=3 if c["nref"] == 3 else 2, **kw)
        return decks2d.plain_k_operator(tb, c["nref"]) if c["nref"] > 3 else tb
    return decks2d.tables(**kw)


@functools.lru_cache(maxsize=None)
def _basin(nx, ny):
    """The tables of a flat basin as a caller with a set-up of their own passes them (exact dispersion at
    3 m, alias mask at half the band, cosine damping zones, nonlinear adjustment over a ramp in x)."""
    x, y = 0.6 * np.arange(nx), 0.6 * np.arange(ny)
    kx, ky = 2 * math.pi * np.fft.fftfreq(nx, 0.6), 2 * math.pi * np.fft.fftfreq(ny, 0.6)
    KX, KY = np.meshgrid(kx, ky)
    K = np.hypot(KX, KY)
    K[0, 0] = 1.0
    c2 = np.where(np.hypot(KX, KY) == 0, G * 3.0, G * np.tanh(3.0 * K) / K)
    mask = ((np.abs(KX) < np.abs(kx).max() / 2) & (np.abs(KY) < np.abs(ky).max() / 2)).astype(float)

    def zone(v):
        d = np.minimum(v - v[0], v[-1] - v) / (0.1 * (v[-1] - v[0]))
        return 0.5 * (1 + np.cos(math.pi * np.minimum(d, 1.0)))

    charac = np.maximum(zone(x)[None, :], zone(y)[:, None]) / 5.0
    chi = np.tile(0.5 * (1 - np.cos(math.pi * np.clip((x - x[nx // 8]) / (x[nx // 4] - x[nx // 8]), 0, 1))), (ny, 1))
    return dict(nx=nx, ny=ny, model=2, propagation=0, cpeak=4.0, kx=kx, ky=ky, c2d=np.sqrt(c2), l2d=c2 * np.where(
        np.hypot(KX, KY) == 0, 0.0, K) ** 2 / G, aal=mask, charac=charac, chiadj=chi)


def _sea2d(tb, Hs, Tp, depth, seed):
    """A short-crested sea that fills the basin (JONSWAP, cos^2s with s = 10 about +x), at rest in the
    damping zones, let down over shallow water; [Re eta^|Im eta^|Re u^|Im u^|Re v^|Im v^]."""
    rng = np.random.default_rng([seed, 13])
    kx, ky = tb["kx"], tb["ky"]
    nx, ny = kx.size, ky.size
    KX, KY = np.meshgrid(kx, ky)
    K = np.maximum(np.hypot(KX, KY), 1e-6)
    w = np.sqrt(G * K * np.tanh(K * depth))
    cg = 0.5 * w / K * (1 + 2 * K * depth / np.sinh(np.minimum(2 * K * depth, 500.0)))
    amp = np.sqrt(_jonswap(w, Hs, Tp, 3.3) * cg / K) * np.cos(0.5 * np.arctan2(KY, KX)) ** 10
    amp[0, 0] = 0.0
    eh = amp * np.exp(2j * math.pi * rng.random((ny, nx)))
    fields = [np.fft.ifft2(eh).real, np.fft.ifft2(eh * G * KX / w).real, np.fft.ifft2(eh * G * KY / w).real]
    win = [np.sin(0.5 * math.pi * np.minimum(1.0, np.minimum(np.arange(n), n - 1 - np.arange(n)) / (0.12 * n))) ** 2
           for n in (ny, nx)]
    shape = win[0][:, None] * win[1][None, :] * Hs / (4 * fields[0].std())
    if "depth" in tb:
        shape = shape * np.minimum(1.0, tb["depth"].reshape(ny, nx) / (6.0 * Hs))
    out = []
    keep = (np.abs(np.fft.fftfreq(nx)) < 1 / 6.5)[None, :] & (np.abs(np.fft.fftfreq(ny)) < 1 / 6.5)[:, None]
    for f in fields:
        s = np.where(keep, np.fft.fft2(f * shape), 0.0)
        out += [s.real.ravel(), s.imag.ravel()]
    return np.concatenate(out)


# ---------------------------------------------------------------------------
# the network's records
# ---------------------------------------------------------------------------
_BAND = np.array([0.6, 0.75, 0.9, 1.0, 1.1, 1.3, 1.6, 2.0])


def _records(n, seed):
    """Training records of n grid points: depths over the four references' range, the dominant band of a
    1.5-3 s sea, smoothed depths near the point's own, the true phase speed as the target."""
    rng = np.random.default_rng([seed, 17])
    D = 0.05 * (2.0 / 0.05) ** (np.arange(4) / 3)
    pos = rng.random(n) * 3
    h = 0.05 * (2.0 / 0.05) ** (pos / 3)
    wp = 2 * math.pi / (1.5 + 1.5 * rng.random(n))
    kd = wp / np.sqrt(G * h) * (1 + 0.1 * wp * wp * h / G)
    kap = kd[:, None] * _BAND[None, :]
    Gm = np.stack([G * np.tanh(kap * d) / kap for d in D], axis=2)
    T = G * np.tanh(kap * h[:, None]) / kap
    f = np.stack([pos - 1.5] + [pos - 1.5 + s * rng.standard_normal(n) for s in (0.05, 0.2, 0.4)] + [np.log(kd * h)],
                 axis=1)
    return np.concatenate([f, Gm.reshape(n, -1), T], axis=1).astype(np.float32)


def _weights(seed):
    rng = np.random.default_rng([seed, 19])
    p = np.zeros(1380, dtype=np.float32)
    off = 0
    for o, i in ((32, 5), (32, 32), (4, 32)):
        a = math.sqrt(6.0 / (o + i))
        p[off:off + o * i] = rng.uniform(-a, a, o * i)
        off += o * i + o
    return p


# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("rhs1d", "step1d", "run1d"):
        c = _full(case)
        paths = _decks(json.dumps(c, sort_keys=True))
        eng = hw.Engine(paths, nref=c["nref"] if c["bottom"] != "flat" else 0, seed=seed, slice=c["slice"], **TOL)
        y = _seas(c, seed)
        if kind != "run1d":
            return dict(kind=kind, eng=eng, y=y[0], work=np.empty_like(y[0]))
        y = _pinned(np.concatenate(y))
        return dict(kind=kind, eng=eng, y=y, out=_pinned(np.zeros_like(y)), i=1, window=c["window"], n=min(eng.nt))
    if kind == "rhs2d":
        tb = _basin(case["nx"], case["ny"])
        return dict(kind=kind, eng=Engine2D(tb, **TOL), y=_sea2d(tb, 0.3, 4.0, 3.0, seed))
    if kind == "run2d":
        tb = _tables(json.dumps({**case, "name": ""}, sort_keys=True))
        big = case["bottom"] == "harbour"
        y = _pinned(_sea2d(tb, 0.25 if big else 0.15, 6.0 if big else 4.0, 5.0 if big else 3.0, seed))
        return dict(kind=kind, eng=Engine2D(tb, **TOL), y=y, out=_pinned(np.zeros_like(y)), t=4.0, h=0.01,
                    window=case["window"])
    return dict(kind=kind, mlp=learned.MLP(), records=_records(case["records"], seed), p0=_weights(seed),
                batch=case["batch"], epochs=case["epochs"])


def run(s):
    kind = s["kind"]
    if kind == "rhs1d":
        return s["eng"].rhs(1.0, s["y"])
    if kind == "rhs2d":
        return s["eng"].rhs(1.0, s["y"])
    if kind == "step1d":
        s["work"][:] = s["y"]
        t, _ = s["eng"].evolve_apply(5.0, 5.5, 2e-3, s["work"])
        return {"t": t, "y": s["work"]}
    if kind == "run1d":
        eng = s["eng"]
        if s["i"] + s["window"] > s["n"]:   # past the influx signal: from its start again
            eng.reset()
            s["i"] = 1
        s["i"] += s["window"]
        eng.set_states(s["y"])
        eng.run(s["i"], sync=False)
        return eng.get_states(s["out"])
    if kind == "run2d":
        eng = s["eng"]
        if s["t"] + s["window"] > 29.9:
            s["t"], s["h"] = 4.0, 0.01
        t1 = s["t"] + s["window"]
        eng.set_state(s["t"], s["h"], s["y"])
        eng.run_to_time(t1)
        s["t"], s["h"] = eng.state_into(s["out"])
        return s["out"]
    s["mlp"].set_params(s["p0"])
    losses = s["mlp"].train(s["records"], epochs=s["epochs"], batch=s["batch"], lr=3e-3)
    return {"losses": losses, "params": s["mlp"].params()}


def work(case):
    """Bytes: states in and out and the operator tables once.  Flops: the transforms that the RHS cannot do
    without (real signals, two to a complex transform of 5 N log2 N) and 40-80 pointwise ones, times the RHS
    evaluations that the tolerances ask of a window."""
    kind = case["kind"]
    if kind == "train":
        n = case["records"]
        return dict(bytes=4.0 * 45 * n, flops=3.0 * 2 * (5 * 32 + 32 * 32 + 32 * 4) * n * case["epochs"])
    if kind in ("rhs1d", "step1d", "run1d"):
        c = _full(case)
        nbytes = flops = 0.0
        for m in range(c["members"]):
            p = _member(c, m)
            N, K = p["nx"], 0 if c["bottom"] == "flat" else c["nref"]
            order = int(c["model"][2])
            hss = 0 if not K or order == 1 else (K + (K + 1) // 2) * (2 if order == 2 else 3)
            ffts = {1: 2, 2: 6, 3: 9}[order] + hss
            kc = math.pi / (p["length"] / N) / (order if order == 3 else 2)
            edge = math.sqrt(G * kc * math.tanh(kc * p["depth"]))
            n_rhs = 1 if kind == "rhs1d" else 7 if kind == "step1d" else RHS_PER_RAD * edge * DT * c["window"]
            nbytes += 8.0 * N * (8 + 9 + 2 * K)
            flops += n_rhs * N * (5.0 * math.log2(N) * ffts + 60 + 8 * K)
        return dict(bytes=nbytes, flops=flops)
    N = case["nx"] * case["ny"]
    if kind == "rhs2d":
        return dict(bytes=8.0 * N * (12 + 5), flops=N * (5.0 * math.log2(N) * 11 + 80))
    big = case["bottom"] == "harbour"
    K = 0 if case["bottom"] == "flat" else case["nref"]
    hss = 0 if not K else (K + (K + 1) // 2) * {1: 2, 2: 4, 3: 8}[case["model"]]
    ffts = {1: 4, 2: 11, 3: 16}[case["model"]] + hss
    kc = math.pi / (300.0 / 1024 if big else 0.6) / {1: 1, 2: 2, 3: 3}[case["model"]]
    n_rhs = RHS_PER_RAD * math.sqrt(G * kc) * case["window"] * (20 if case["breaking"] else 1)
    return dict(bytes=8.0 * N * (12 + 6 + 3 * K), flops=n_rhs * N * (5.0 * math.log2(N) * ffts + 80 + 16 * K))


# ---------------------------------------------------------------------------
# 64-bit values in plain numpy
# ---------------------------------------------------------------------------
def _freqspace(length, n):
    d0 = 2 * math.pi / length
    lo = -0.5 * 2 * math.pi / (length / (n - 1))
    hi = -lo - d0
    d = (hi - lo) / (n - 1)
    i = np.arange(n // 2)
    return np.concatenate([lo + (n // 2 + i) * d, lo + i * d])


def _exact_rhs1d(c, y):
    """rhs_HsF1 / rhs_HsF2 on a flat bottom without influx: linear part, second-order products, damping, mask."""
    p = _member(c, 0)
    N, L, h = p["nx"], p["length"], p["depth"]
    order = int(c["model"][2])
    k = _freqspace(L, N)
    with np.errstate(divide="ignore", invalid="ignore"):
        c2 = np.where(k == 0, G * h, G * np.tanh(k * h) / k)
    x = np.arange(N) * (L / (N - 1))
    w = 0.05 * L

    def side(d):   # 1 in the water, falling to 0 over the damping zone
        return 0.5 * (1 - np.cos(math.pi * np.clip(d / w, 0.0, 1.0)))

    char = 1 - side(x) * side(L - x)
    damp = 7 * math.sqrt(G * h) / (0.9 * w) * char
    k0 = k[N // (2 if order == 1 else 4) - 1]
    with np.errstate(divide="ignore", invalid="ignore"):
        mask = ((k0 - np.abs(k)) / np.abs(k0 - np.abs(k)) + 1) / 2
    mask[N // (2 if order == 1 else 4) - 1] = 0.5
    e, u = y[:N] + 1j * y[N:2 * N], y[2 * N:3 * N] + 1j * y[3 * N:]
    F, R = np.fft.fft, lambda a: np.fft.ifft(a).real
    pe, pu = R(e), R(u)
    de, du = -1j * k * c2 / G * u - F(damp * pe), -1j * k * G * e - F(damp * pu)
    if order == 2:
        m0 = R(-1j * k * c2 / G * u)
        de += F(R(-k * k * c2 / G * F(pe * m0) - 1j * k * F(pe * pu)))   # the adjustment keeps real fields
        du += F(R(-0.5j * k * F(pu * pu - m0 * m0)))
    de, du = de * mask, du * mask
    return np.concatenate([de.real, de.imag, du.real, du.imag])


def _sym2d(a):
    """fftwcomplex_2d_sym: the right half and the lower left column from the mirror, self-conjugate points real."""
    ny, nx = a.shape
    a = a.copy()
    m = np.conj(np.roll(a[::-1, ::-1], (1, 1), (0, 1)))
    a[:, nx // 2 + 1:] = m[:, nx // 2 + 1:]
    a[ny // 2 + 1:, 0] = m[ny // 2 + 1:, 0]
    for i in (0, ny // 2):
        for j in (0, nx // 2):
            a[i, j] = a[i, j].real
    return a


def _exact_rhs2d(tb, y):
    """rhs_AB2_2DF_uv without a source."""
    ny, nx = tb["ny"], tb["nx"]
    z = y.reshape(3, 2, ny, nx)
    e, u, v = (z[f, 0] + 1j * z[f, 1] for f in range(3))
    kx, ky = tb["kx"][None, :], tb["ky"][:, None]
    cg, L = tb["c2d"] ** 2 / G, tb["l2d"]
    damp = 7 * tb["cpeak"] * tb["charac"]
    F, R = np.fft.fft2, lambda a: np.fft.ifft2(_sym2d(a)).real
    mu, mv = -1j * cg * kx * u, -1j * cg * ky * v
    pe, pu, pv, pmu, pmv, pl = R(e), R(u), R(v), R(mu), R(mv), R(mu + mv)
    dH = F(0.5 * (pu * pu + pv * pv - pl * pl))
    adj = lambda a: F(tb["chiadj"] * np.fft.ifft2(_sym2d(a)))  # noqa: E731
    de = mu + mv + adj(-L * F(pe * pmu) - 1j * kx * F(pe * pu)) + adj(-L * F(pe * pmv) - 1j * ky * F(pe * pv))
    de -= F(damp * pe)
    du = -1j * G * kx * e - adj(1j * kx * dH) - F(damp * pu)
    dv = -1j * G * ky * e - adj(1j * ky * dH) - F(damp * pv)
    return np.concatenate([part.ravel() for d in (de, du, dv) for part in ((d * tb["aal"]).real, (d * tb["aal"]).imag)])


def _exact_train(recs, p0, batch, epochs, lr=3e-3):
    """The network's forward, backward and Adam."""
    recs, p = recs.astype(np.float64), p0.astype(np.float64)
    cut = np.cumsum([160, 32, 1024, 32, 128])
    m1, m2, losses, step = np.zeros_like(p), np.zeros_like(p), [], 0
    for _ in range(epochs):
        total = 0.0
        for off in range(0, len(recs), batch):
            r = recs[off:off + batch]
            x, Gm, T = r[:, :5], r[:, 5:37].reshape(-1, 8, 4), r[:, 37:]
            W1, b1, W2, b2, W3, b3 = np.split(p, cut)
            W1, W2, W3 = W1.reshape(32, 5), W2.reshape(32, 32), W3.reshape(4, 32)
            h1 = np.tanh(x @ W1.T + b1)
            h2 = np.tanh(h1 @ W2.T + b2)
            q = h2 @ W3.T + b3
            q = np.exp(q - q.max(axis=1, keepdims=True))
            q /= q.sum(axis=1, keepdims=True)
            err = (np.einsum("nmj,nj->nm", Gm, q) - T) / T
            total += float((err ** 2).mean(axis=1).sum())
            dw = np.einsum("nm,nmj->nj", 2 * err / (8 * T), Gm)
            dz = q * (dw - (q * dw).sum(axis=1, keepdims=True))
            d2 = dz @ W3 * (1 - h2 * h2)
            d1 = d2 @ W2 * (1 - h1 * h1)
            g = np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), (dz.T @ h2).ravel(),
                                dz.sum(0)]) / len(r)
            step += 1
            m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
            p = p - lr * (m1 / (1 - 0.9 ** step)) / (np.sqrt(m2 / (1 - 0.999 ** step)) + 1e-8)
        losses.append(total / len(recs))
    return {"losses": np.array(losses), "params": p}


def exact(case, seed):
    """None for the steps and runs: which steps are accepted is the integrator's own answer."""
    if case["kind"] == "rhs1d":
        c = _full(case)
        return _exact_rhs1d(c, _seas(c, seed)[0])
    if case["kind"] == "rhs2d":
        tb = _basin(case["nx"], case["ny"])
        return _exact_rhs2d(tb, _sea2d(tb, 0.3, 4.0, 3.0, seed))
    if case["kind"] == "train":
        return _exact_train(_records(case["records"], seed), _weights(seed), case["batch"], case["epochs"])
    return None
