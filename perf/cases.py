"""Timed cases of the trajectory and transport-statistics path.

Each case is one call, or the few calls, that a user's program makes through
the Python host: pushing device-resident ensembles (FastEnsemble,
DeviceEnsemble), whole host-state runs (run_push_host), a set of campaigns in
a Batch, and the lag statistics over mu caches and phase-space caches.  The
sizes are those of the repository's own configurations and benchmark, or
generic ones between them.

listed() and draw() give the cases, prepare() what a program holds before the
call (fields, states, caches, accumulators, on the GPU), run() one pass,
work() the bytes and operations that a pass cannot do without, and exact()
the outputs in 64 bits from plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from particle_transport_b200 import runner as R
from particle_transport_b200 import stats as S
from particle_transport_b200.batch import Batch
from particle_transport_b200.fields import FieldLibrary, build_uniform_grid
from particle_transport_b200.time_units import build_mu_edges_full, log_spaced_lag_steps

C = 2.99792458e8
QE = 1.602176634e-19
MP = 1.67262192369e-27
B0_T = 1e-10  # 1 microgauss
KEYS = ("x1", "x2", "x3", "p1", "p2", "p3")
DEV = "cuda"


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the smallest campaign (64^3, 4096 protons, 1 GeV): one gyroperiod of the FP32 push over FP32
        # bricks, mu rows every 4 steps; launches and the latency of a step count
        {"name": "push_small", "kind": "push32", "storage": "brick_f32", "grid": 64, "n": 4096, "energy": 1.0,
         "steps": 64, "spg": 64, "stride": 4, "sort_every": 0, "pitch": 0, "cache": "mu", "periodic": True,
         "db": 0.5},
        # the large single campaign: 512^3 BF16 bricks, 16.7M protons at 10 GeV, re-sorted every 64 steps,
        # time-fastest mu cache every 8 steps
        {"name": "push_large_bf16", "kind": "push32", "storage": "brick_bf16", "grid": 512, "n": 16777216,
         "energy": 10.0, "steps": 64, "spg": 64, "stride": 8, "sort_every": 64, "pitch": 8, "cache": "mu",
         "periodic": True, "db": 1.0},
        # an ordinary campaign of fast particles (100 GeV cross a brick in about two steps) over FP32 bricks,
        # with a ragged particle count
        {"name": "push_fast_particles_f32", "kind": "push32", "storage": "brick_f32", "grid": 256, "n": 1000003,
         "energy": 100.0, "steps": 64, "spg": 128, "stride": 8, "sort_every": 16, "pitch": 8, "cache": "mu",
         "periodic": True, "db": 0.5},
        # the FP64 push (bit-exact form) over FP64 bricks, brick-sorted, mu rows
        {"name": "push_f64_brick", "kind": "push64", "storage": "brick_f64", "grid": 256, "n": 1048576,
         "energy": 1.0, "steps": 64, "spg": 128, "stride": 8, "sort_every": 64, "cache": "mu", "periodic": True,
         "db": 0.5},
        # the default of the ensemble runners: FP64 push over the reference field layout, host state,
        # phase-space rows handed to the writer; open boundary, particles leave the box
        {"name": "run_host_f64_phase_space", "kind": "host", "storage": "ref_f64", "grid": 128, "n": 65536,
         "energy": 10.0, "nsteps": 257, "spg": 64, "stride": 8, "sort_every": 0, "cache": "phase_space",
         "periodic": False, "db": 0.5},
        # a whole host-state run of the FP32 push with mu rows handed to the writer
        {"name": "run_host_bf16_mu", "kind": "host", "storage": "brick_bf16", "grid": 256, "n": 1000000,
         "energy": 10.0, "nsteps": 257, "spg": 128, "stride": 8, "sort_every": 64, "cache": "mu",
         "periodic": True, "db": 0.5},
        # campaigns of uneven sizes and energies (1, 10, 100 GeV) admitted to one batch, run to their end,
        # read back and removed: what a batched run or a serving loop does
        {"name": "batch_campaigns", "kind": "batch", "storage": "brick_f32", "grid": 256, "n": 2000000, "camps": 6,
         "steps": 256, "spg": 64, "stride": 8, "db": 0.5},
        # D_mumu of the large campaign: 4001 saves, log-spaced lags up to the whole series, 50 |mu| bins
        {"name": "dmumu_large", "kind": "dmumu", "n": 131072, "nsave": 4001, "lags": 64, "bins": 50,
         "mode": "sliding", "abs": True, "tf": True, "dead": 0.0},
        # D_mumu of the smallest campaign, from mu rows
        {"name": "dmumu_small", "kind": "dmumu", "n": 4096, "nsave": 801, "lags": 20, "bins": 20,
         "mode": "sliding", "abs": True, "tf": False, "dead": 0.0},
        # injection estimator with signed bins; some particles left an open box
        {"name": "dmumu_injection", "kind": "dmumu", "n": 524287, "nsave": 801, "lags": 32, "bins": 40,
         "mode": "injection", "abs": False, "tf": False, "dead": 0.2},
        # D_mumu from a phase-space cache (mu reconstructed at the Float32 compute precision)
        {"name": "dmumu_phase_space", "kind": "dmumu_ps", "grid": 256, "n": 65536, "nsave": 801, "lags": 32,
         "bins": 20, "mode": "sliding", "energy": 10.0},
        # momentum products of a phase-space subset: D_pp on log-spaced lags, 16 energy snapshots and their
        # 256-bin histograms
        {"name": "dpp_energies", "kind": "dpp", "n": 65536, "nsave": 4001, "lags": 64, "snaps": 16, "hist": 256,
         "dead": 0.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["push32", "push32", "push64", "host", "batch", "dmumu", "dmumu", "dmumu_ps", "dpp"])
    grid = rng.choice([48, 64, 96, 100, 128, 192, 250, 256])
    if kind in ("push32", "push64", "host"):
        c = {"kind": kind, "storage": rng.choice(["brick_f32", "brick_bf16"]), "grid": grid, "n": 0,
             "energy": math.exp(rng.uniform(0.0, math.log(300.0))), "spg": rng.choice([64, 128]),
             "stride": rng.choice([1, 3, 4, 8, 16]), "sort_every": rng.choice([0, 16, 64]),
             "cache": rng.choice(["mu", "mu", "phase_space"]), "periodic": kind != "host" or rng.random() < 0.5,
             "db": rng.choice([0.5, 1.0])}
        if kind == "push32":
            c["n"] = _log(rng, 1000, 4000000 if c["cache"] == "mu" else 1000000)
            c["steps"] = c["stride"] * _log(rng, max(1, 16 // c["stride"]), max(1, 96 // c["stride"]))
            c["pitch"] = c["steps"] // c["stride"] if c["cache"] == "mu" and rng.random() < 0.5 else 0
            if grid >= 250 and rng.random() < 0.3:
                c["grid"], c["storage"] = 512, "brick_bf16"
        elif kind == "push64":
            c["storage"] = rng.choice(["brick_f64", "ref_f64"])
            c["n"] = _log(rng, 1000, 1000000 if c["storage"] == "brick_f64" else 300000)
            c["steps"] = c["stride"] * _log(rng, max(1, 16 // c["stride"]), max(1, 64 // c["stride"]))
        else:
            c["storage"] = rng.choice(["ref_f64", "brick_f64", "brick_f32", "brick_bf16"])
            c["n"] = _log(rng, 1000, 60000 if c["storage"] == "ref_f64" else 500000)
            if c["cache"] == "phase_space":
                c["n"] = min(c["n"], 100000)
            c["nsteps"] = _log(rng, 50, 400)
            c["stride"] = max(4, c["stride"])
        return c
    if kind == "batch":
        return {"kind": kind, "storage": rng.choice(["brick_f32", "brick_bf16"]), "grid": grid,
                "n": _log(rng, 20000, 2000000), "camps": rng.randint(1, 10), "steps": 64 * rng.randint(1, 4),
                "spg": 64, "stride": rng.choice([4, 8]), "db": 0.5}
    if kind == "dmumu":
        nsave = _log(rng, 60, 6000)
        return {"kind": kind, "n": max(1, min(_log(rng, 500, 400000), 400000000 // nsave)), "nsave": nsave,
                "lags": rng.randint(7, 64), "bins": rng.choice([10, 20, 24, 40, 50]),
                "mode": rng.choice(["sliding", "sliding", "injection"]), "abs": rng.random() < 0.7,
                "tf": rng.random() < 0.5, "dead": rng.choice([0.0, 0.0, 0.1, 0.5])}
    if kind == "dmumu_ps":
        nsave = _log(rng, 60, 2000)
        return {"kind": kind, "grid": min(grid, 192), "n": max(1, min(_log(rng, 500, 200000), 40000000 // nsave)),
                "nsave": nsave, "lags": rng.randint(7, 64), "bins": rng.choice([10, 20, 50]),
                "mode": rng.choice(["sliding", "sliding", "injection"]),
                "energy": math.exp(rng.uniform(0.0, math.log(300.0)))}
    nsave = _log(rng, 60, 6000)
    return {"kind": kind, "n": max(1, min(_log(rng, 500, 300000), 200000000 // nsave)), "nsave": nsave,
            "lags": rng.randint(7, 64), "snaps": rng.randint(2, 16), "hist": rng.choice([64, 100, 256]),
            "dead": rng.choice([0.0, 0.0, 0.1])}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _solenoidal(n, rms, g):
    """Divergence-free Gaussian field, isotropic k^(-11/3) modes 2 <= |k| <= n/2, scaled to rms."""
    k = torch.fft.fftfreq(n, d=1.0 / n, device=DEV)
    kh = torch.fft.rfftfreq(n, d=1.0 / n, device=DEV)
    kz, ky, kx = k.view(n, 1, 1), k.view(1, n, 1), kh.view(1, 1, -1)
    k2 = (kx * kx + ky * ky + kz * kz).clamp_min(1e-20)
    amp = torch.where((k2 >= 4) & (k2 <= (n / 2) ** 2), k2 ** (-11.0 / 12.0), torch.zeros_like(k2))
    a = [torch.complex(torch.randn(amp.shape, generator=g, device=DEV) * amp,
                       torch.randn(amp.shape, generator=g, device=DEV) * amp) for _ in range(3)]
    dot = (kx * a[0] + ky * a[1] + kz * a[2]) / k2
    out = []
    for i, kk in enumerate((kx, ky, kz)):
        out.append(torch.fft.irfftn(a[i] - kk * dot, s=(n, n, n)))
        a[i] = None
    s = rms / math.sqrt(sum(float((f * f).mean()) for f in out))
    return [f.double() * s for f in out]


def _fields(c, g):
    """Six SI components (Bx, By, Bz, ux, uy, uz): B0 along z plus turbulence, u_rms = 1e-4 c."""
    b = _solenoidal(c["grid"], c.get("db", 0.5) * B0_T, g)
    b[2] = b[2] + B0_T
    return b + _solenoidal(c["grid"], 1e-4 * C, g)


def _gamma(energy):
    return energy * 1e9 * QE / (MP * C * C) + 1.0


def _p(energy):
    return math.sqrt(_gamma(energy) ** 2 - 1.0) * MP * C


def _grid(c):
    """Box whose cell is the gyroradius of a 1 GeV proton in B0."""
    return build_uniform_grid(_p(1.0) / (QE * B0_T) * (c["grid"] - 1), c["grid"], c["grid"], c["grid"])


def _dt(energy, spg):
    return 2.0 * math.pi * _gamma(energy) * MP / (QE * B0_T) / spg


def _particles(n, grid, energy, g):
    """Uniform positions, isotropic momenta."""
    r = torch.rand((5, n), generator=g, device=DEV, dtype=torch.float64)
    z = 2.0 * r[3] - 1.0
    phi = 2.0 * math.pi * r[4]
    perp = torch.sqrt((1.0 - z * z).clamp_min(0.0))
    p = _p(energy)
    return {"x1": r[0] * (grid.xmax - grid.xmin) + grid.xmin, "x2": r[1] * (grid.ymax - grid.ymin) + grid.ymin,
            "x3": r[2] * (grid.zmax - grid.zmin) + grid.zmin, "p1": p * perp * torch.cos(phi),
            "p2": p * perp * torch.sin(phi), "p3": p * z}


def _mu_series(c, g):
    """Pitch-angle cosines of particles that scatter: mu = cos(theta), theta a random walk of about 0.05 rad per
    save (the walk is summed in whole numbers, so that the same seed gives the same bits); particles that died
    are NaN from some save on.  Float32 (n, nsave)."""
    n, ns = c["n"], c["nsave"]
    step = (torch.randn((n, ns), generator=g, device=DEV) * 3276.8).round_().to(torch.int32)
    step[:, 0] = torch.randint(0, 205887, (n,), generator=g, device=DEV, dtype=torch.int32)  # theta in [0, pi)
    mu = torch.cos(torch.cumsum(step, dim=1, dtype=torch.int64).to(torch.float32).mul_(1.0 / 65536.0))
    return _kill(mu, c, g)


def _kill(v, c, g):
    if c["dead"] > 0:
        at = torch.randint(0, c["nsave"], (c["n"],), generator=g, device=DEV)
        at[torch.rand(c["n"], generator=g, device=DEV) >= c["dead"]] = c["nsave"]
        v[torch.arange(c["nsave"], device=DEV)[None, :] >= at[:, None]] = math.nan
    return v


def _phase_space(c, grid, g):
    """Positions on straight, periodically wrapped paths and momenta of constant magnitude whose pitch angle walks
    and whose phase turns, Float32 (nsave, 6, n): what a phase-space cache holds, save by save."""
    n, ns = c["n"], c["nsave"]
    r = torch.rand((6, n), generator=g, device=DEV)
    ps = torch.empty((ns, 6, n), dtype=torch.float32, device=DEV)
    theta = torch.acos(2.0 * r[3] - 1.0)
    phase = 2.0 * math.pi * r[4]
    adv = 8.0 * C * _dt(c["energy"], 64) / grid.dx  # cells per save at the speed of light
    x = [r[i] * (c["grid"] - 1) for i in range(3)]
    p = _p(c["energy"])
    for s in range(ns):
        st, ct = torch.sin(theta), torch.cos(theta)
        u = (st * torch.cos(phase), st * torch.sin(phase), ct)
        for k in range(3):
            ps[s, k] = (x[k] * grid.dx).clamp_(grid.xmin, grid.xmax)
            ps[s, 3 + k] = u[k] * p
            x[k] = torch.remainder(x[k] + u[k] * adv, float(c["grid"] - 1))
        theta = theta + 0.05 * torch.randn(n, generator=g, device=DEV)
        phase = phase + math.pi / 4
    return ps


def _momenta(c, g):
    """Float32 momenta (nsave, 3, n) whose magnitude walks by 1e-4 per save around that of 10 GeV."""
    n, ns = c["n"], c["nsave"]
    step = (torch.randn((ns, n), generator=g, device=DEV) * 64.0).round_().to(torch.int32)
    mag = _kill((1.0 + torch.cumsum(step, dim=0, dtype=torch.int64).to(torch.float64) * (1e-4 / 64.0)).t(), c, g).t()
    z = 2.0 * torch.rand((ns, n), generator=g, device=DEV) - 1.0
    phi = 2.0 * math.pi * torch.rand((ns, n), generator=g, device=DEV)
    perp = torch.sqrt((1.0 - z * z).clamp_min(0.0))
    out = torch.empty((ns, 3, n), dtype=torch.float32, device=DEV)
    mag = mag * _p(10.0)
    out[:, 0] = (mag * (perp * torch.cos(phi))).float()
    out[:, 1] = (mag * (perp * torch.sin(phi))).float()
    out[:, 2] = (mag * z).float()
    return out


def _lags(c):
    return log_spaced_lag_steps(c["nsave"] - 1, c["lags"])


def _edges(c):
    return build_mu_edges_full(0.0, 1.0, c["bins"], bin_abs=bool(c.get("abs", True)))[0]


def _camps(c):
    """Sizes, energies and re-sort cadences (in epochs of 16 steps) of a batch's campaigns: sizes spread by a factor
    of about 16 over the campaigns."""
    w = [2.0 ** (4.0 * i / max(1, c["camps"] - 1)) for i in range(c["camps"])]
    ns = [max(1, int(c["n"] * v / sum(w))) for v in w]
    return [(n, (1.0, 10.0, 100.0)[i % 3], (4, 4, 1)[i % 3]) for i, n in enumerate(ns)]


def _cache(c, n, rows):
    if c["cache"] == "phase_space":
        return torch.zeros((rows, 6, n), dtype=torch.float32, device=DEV)
    return torch.zeros((n, c["pitch"]) if c.get("pitch") else (rows, n), dtype=torch.float32, device=DEV)


def prepare(case, seed):
    c, g = dict(case), _gen(seed)
    kind = c["kind"]
    s = {"c": c}
    if kind in ("push32", "push64", "host", "batch", "dmumu_ps"):
        grid = s["grid"] = _grid(c)
        raw = _fields(c, g)
    if kind in ("push32", "push64", "host", "batch"):
        s["field"] = FieldLibrary(raw, grid, c["storage"], B_ref_T=B0_T)
        del raw
    if kind in ("push32", "push64"):
        state = _particles(c["n"], grid, c["energy"], g)
        alive = torch.ones(c["n"], dtype=torch.uint8, device=DEV)
        s["ens"] = (R.FastEnsemble if kind == "push32" else R.DeviceEnsemble)(s["field"], state, alive)
        s["rows"] = (c["steps"] + c["stride"] - 1) // c["stride"]
        s["cache"] = _cache(c, c["n"], s["rows"])
        s["params"] = R.push_params(_dt(c["energy"], c["spg"]), 1 << 40, c["stride"], c["periodic"], c["cache"],
                                    precision="f32" if kind == "push32" else "f64", sort_every=c["sort_every"],
                                    cache_pitch=c.get("pitch", 0))
        s["step"] = 0
    elif kind == "host":
        state = _particles(c["n"], grid, c["energy"], g)
        s["initial"] = {k: v.cpu().numpy() for k, v in state.items()}
        f64 = c["storage"] in ("ref_f64", "brick_f64")
        s["params"] = R.push_params(_dt(c["energy"], c["spg"]), c["nsteps"], c["stride"], c["periodic"], c["cache"],
                                    precision="f64" if f64 else "f32", sort_every=c["sort_every"])
        s["rows"] = R.CacheCollector(c["n"], R.n_saves(c["nsteps"], c["stride"]), c["cache"])
    elif kind == "batch":
        s["batch"] = Batch(c["n"] + 64, max_campaigns=c["camps"], storage=c["storage"], steps_per_epoch=16)
        s["camps"] = []
        for n, energy, sort in _camps(c):
            s["camps"].append({"state": _particles(n, grid, energy, g), "dt": _dt(energy, c["spg"]), "sort": sort,
                               "cache": torch.zeros((n, R.n_saves(c["steps"] + 1, c["stride"])), device=DEV)})
    elif kind == "dmumu":
        mu = _mu_series(c, g)
        s["mu"] = mu if c["tf"] else mu.t().contiguous()
    elif kind == "dmumu_ps":
        s["B"] = [b.float() for b in raw[:3]]
        s["ps"] = _phase_space(c, grid, g)
    else:
        s["mom"] = _momenta(c, g)
        s["p0"] = _p(10.0)
        s["at"] = np.linspace(0, c["nsave"] - 1, c["snaps"]).round().astype(np.int64)
        s["acc"] = S.new_dpp_accumulators(len(_lags(c)), device=DEV)
        s["energy"] = torch.zeros((c["n"], c["snaps"]), dtype=torch.float64, device=DEV)
        s["hist"] = torch.zeros((c["snaps"], c["hist"]), dtype=torch.int64, device=DEV)
    if kind in ("dmumu", "dmumu_ps", "dpp"):
        s["lags"] = _lags(c)
    if kind in ("dmumu", "dmumu_ps"):
        s["edges"] = _edges(c)
        s["acc"] = S.new_dmumu_accumulators(len(s["lags"]), c["bins"], device=DEV)
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind in ("push32", "push64"):
        # the next segment of a trajectory: its steps, its cache rows, the state after it
        first = -(-s["step"] // c["stride"])
        rows = -(-(s["step"] + c["steps"]) // c["stride"]) - first
        s["ens"].advance(s["params"], s["step"], c["steps"], s["cache"], first, rows)
        s["step"] += c["steps"]
        if kind == "push32":
            state, alive = s["ens"].export()
        else:
            state, alive = s["ens"].state, s["ens"].alive
        return {"cache": s["cache"], "alive": alive, **state}
    if kind == "host":
        # the run advances its host state in place: it gets its own copy of the initial one, as the runners do
        state = {k: v.copy() for k, v in s["initial"].items()}
        alive = np.ones(c["n"], dtype=np.uint8)
        count = R.run_push_host(s["field"], state, alive, s["params"], s["rows"])
        out = {"count": count, "alive": alive, **state}
        if c["cache"] == "mu":
            out["mu"] = s["rows"].mu
        else:
            out["positions"], out["momenta"] = s["rows"].positions, s["rows"].momenta
        return out
    if kind == "batch":
        b = s["batch"]
        ids = [b.add(s["field"], k["state"], k["dt"], c["steps"] + 1, c["stride"], cache=k["cache"],
                     sort_every=k["sort"], time_fastest=True) for k in s["camps"]]
        b.run(c["steps"] // 16 + 1)
        out = []
        for i, k in zip(ids, s["camps"]):
            state, _ = b.export(i)
            out.append({"mu": k["cache"], "x": torch.stack([state[q] for q in KEYS[:3]]),
                        "p": torch.stack([state[q] for q in KEYS[3:]])})
            b.remove(i)
        return out
    a = s["acc"]
    if kind == "dpp":
        S.process_momenta_chunk_dpp(s["mom"], s["lags"], s["p0"], a["counts"], a["sum_delta_p"], a["sum_delta_p2"],
                                    a["sum_delta_p_norm"], a["sum_delta_p_norm2"])
        S.fill_energy_snapshots(s["energy"], s["mom"], s["at"])
        S.energy_histogram(s["mom"], s["at"], 1.0, 100.0, c["hist"], s["hist"])
        return {"energy": s["energy"], "hist": s["hist"], **a}
    acc = (a["particle_counts"], a["particle_means"], a["particle_m2s"], a["pair_sum_squares"], a["pair_counts"],
           a["dmumu_counts"], a["dmumu_sum_delta"], a["dmumu_sum_delta2"])
    if kind == "dmumu":
        S.process_mu_chunk_dmumu(s["mu"], s["lags"], s["edges"], *acc, start_mode=c["mode"], bin_abs=c["abs"],
                                 layout="time_fastest" if c["tf"] else "particle_fastest")
    else:
        S.process_phase_space_chunk_dmumu(s["ps"][:, 0:3], s["ps"][:, 3:6], *s["B"], s["grid"], s["lags"],
                                          s["edges"], *acc, start_mode=c["mode"])
    return dict(a)


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
NODE = {"brick_f32": 24, "brick_bf16": 12, "brick_f64": 48, "ref_f64": 48}
PUSH_FLOPS = 42 * 3 + 110  # six components by seven lerps, then the Boris step and the drift


def _starts(c):
    """Pairs of one particle over all lags."""
    ls = [int(v) for v in _lags(c)]
    return len(ls) if c.get("mode") == "injection" else sum(c["nsave"] - v for v in ls)


def work(case):
    c = dict(case)
    kind = c["kind"]
    if kind in ("push32", "push64"):
        rows = (c["steps"] + c["stride"] - 1) // c["stride"]
        row = 4 if c["cache"] == "mu" else 24
        # state in and out (49 bytes a particle in either precision), the cache, the field that the particles touch
        field = NODE[c["storage"]] * min(c["grid"] ** 3, 8 * c["n"] * c["steps"])
        return {"bytes": c["n"] * (2 * 49 + rows * row) + field, "flops": c["n"] * c["steps"] * PUSH_FLOPS}
    if kind == "host":
        rows = R.n_saves(c["nsteps"], c["stride"])
        row = 4 if c["cache"] == "mu" else 24
        field = NODE[c["storage"]] * min(c["grid"] ** 3, 8 * c["n"] * c["nsteps"])
        return {"bytes": c["n"] * (2 * 49 + rows * row) + field, "flops": c["n"] * (c["nsteps"] - 1) * PUSH_FLOPS}
    if kind == "batch":
        n = sum(v[0] for v in _camps(c))
        rows = R.n_saves(c["steps"] + 1, c["stride"])
        return {"bytes": n * (2 * 49 + rows * 4) + NODE[c["storage"]] * min(c["grid"] ** 3, 8 * n * c["steps"]),
                "flops": n * c["steps"] * PUSH_FLOPS}
    if kind == "dmumu":
        # the injection estimator needs the first save and the lags' saves only
        per = 4 * (1 + len(_lags(c))) if c["mode"] == "injection" else 4 * c["nsave"]
        return {"bytes": c["n"] * per, "flops": c["n"] * _starts(c) * 4}
    if kind == "dmumu_ps":
        saves = 1 + len(_lags(c)) if c["mode"] == "injection" else c["nsave"]
        return {"bytes": c["n"] * 24 * saves + 12 * min(c["grid"] ** 3, 8 * c["n"] * saves),
                "flops": c["n"] * (saves * 100 + _starts(c) * 4)}
    return {"bytes": c["n"] * (12 * c["nsave"] + 8 * c["snaps"]), "flops": c["n"] * (_starts(c) * 4 + 6 * c["nsave"])}


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------
def _corner_fields(raw):
    return torch.stack([f.reshape(-1) for f in raw], dim=1)


def _interpolate(table, x, grid, n):
    idx, t = [], []
    for q in range(3):
        f = (x[q] - grid.xmin) / grid.dx
        i = f.floor().clamp(0, n - 2)
        idx.append(i.long())
        t.append((f - i).unsqueeze(1))
    out = 0.0
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                w = ((t[0] if dx else 1 - t[0]) * (t[1] if dy else 1 - t[1]) * (t[2] if dz else 1 - t[2]))
                out = out + w * table[idx[0] + dx + n * (idx[1] + dy + n * (idx[2] + dz))]
    return out


def _cross(a, b):
    return torch.stack([a[:, 1] * b[:, 2] - a[:, 2] * b[:, 1], a[:, 2] * b[:, 0] - a[:, 0] * b[:, 2],
                        a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]], dim=1)


def _push(c, grid, table, state, dt, steps, samples, periodic, want):
    """`steps` relativistic Boris steps in 64 bits; rows at samples 0, stride, ... below `samples`."""
    n = c["grid"]
    x = [state[k].clone() for k in KEYS[:3]]
    p = torch.stack([state[k] for k in KEYS[3:]], dim=1)
    alive = torch.ones(p.shape[0], dtype=torch.bool, device=DEV)
    rows, width = [], grid.xmax - grid.xmin
    for s in range(samples):
        last = s >= steps
        save = s % c["stride"] == 0
        if last and not save:
            continue
        f = _interpolate(table, x, grid, n)
        b, u = f[:, :3], f[:, 3:]
        if save:
            if want == "mu":
                v = ((p * b).sum(1) / (p.norm(dim=1) * b.norm(dim=1))).clamp(-1.0, 1.0)
                rows.append(torch.where(alive, v, math.nan))
            else:
                v = torch.cat([torch.stack(x), p.t()])
                rows.append(torch.where(alive, v, math.nan))
        if last:
            continue
        kick = -_cross(u, b) * (QE * dt / 2.0)
        pm = p + kick
        gm = torch.sqrt(1.0 + (pm * pm).sum(1, keepdim=True) / (MP * C) ** 2)
        t = b * (QE * dt / (2.0 * MP)) / gm
        sv = 2.0 * t / (1.0 + (t * t).sum(1, keepdim=True))
        pn = pm + _cross(pm + _cross(pm, t), sv) + kick
        gn = torch.sqrt(1.0 + (pn * pn).sum(1, keepdim=True) / (MP * C) ** 2)
        v = pn / (gn * MP)
        p = torch.where(alive[:, None], pn, p)
        for q in range(3):
            xn = x[q] + v[:, q] * dt
            if periodic:
                xn = xn - torch.floor((xn - grid.xmin) / width) * width
            x[q] = torch.where(alive, xn, x[q])
        if not periodic:
            for q in range(3):
                alive = alive & (x[q] >= grid.xmin) & (x[q] <= grid.xmax)
    return x, p, rows


def _push_all(c, grid, table, state, dt, steps, samples, periodic, want):
    parts = []
    n = state["x1"].shape[0]
    for i in range(0, n, 1 << 20):
        sub = {k: v[i:i + (1 << 20)] for k, v in state.items()}
        parts.append(_push(c, grid, table, sub, dt, steps, samples, periodic, want))
    x = [torch.cat([q[0][k] for q in parts]) for k in range(3)]
    p = torch.cat([q[1] for q in parts])
    rows = torch.stack([torch.cat([q[2][r] for q in parts], dim=-1) for r in range(len(parts[0][2]))])
    return x, p, rows


def _follows(c, energy, steps):
    """Whether a trajectory of this length still follows the 64-bit one: a stored FP32 or BF16 field differs from the
    field by its rounding, and in turbulence two trajectories part exponentially (the faster, the wider their
    orbits)."""
    if c["storage"] in ("ref_f64", "brick_f64"):
        return True
    return steps <= c["spg"] * (2 if c["storage"] == "brick_bf16" and energy <= 30.0 else 4 if energy <= 30.0 else 1)


def _exact_push(c, seed):
    g = _gen(seed)
    grid = _grid(c)
    table = _corner_fields(_fields(c, g))
    host = c["kind"] == "host"
    if c["kind"] == "batch":
        out = []
        for n, energy, _ in _camps(c):
            state = _particles(n, grid, energy, g)
            if not _follows(c, energy, c["steps"]):
                out.append(None)
                continue
            x, p, rows = _push_all(c, grid, table, state, _dt(energy, c["spg"]), c["steps"], c["steps"] + 1, True, "mu")
            out.append({"mu": rows.t(), "x": torch.stack(x), "p": p.t()})
        return out
    state = _particles(c["n"], grid, c["energy"], g)
    steps = c["nsteps"] - 1 if host else c["steps"]
    samples = c["nsteps"] if host else c["steps"]
    x, p, rows = _push_all(c, grid, table, state, _dt(c["energy"], c["spg"]), steps, samples, c["periodic"], c["cache"])
    out = {"alive": None, **dict(zip(KEYS[:3], x)), **{k: p[:, i].contiguous() for i, k in enumerate(KEYS[3:])}}
    if not host:
        out["cache"] = rows.t().contiguous() if c.get("pitch") else rows
    elif c["cache"] == "mu":
        out["count"], out["mu"] = None, rows
    else:
        out["count"], out["positions"], out["momenta"] = None, rows[:, :3].contiguous(), rows[:, 3:].contiguous()
    return out


def _exact_mu(c, seed):
    """mu (n, nsave) in 64 bits."""
    g = _gen(seed)
    if c["kind"] == "dmumu":
        return _mu_series(c, g)
    grid = _grid(c)
    raw = _fields(c, g)
    table = _corner_fields([b.float().double() for b in raw[:3]])
    ps = _phase_space(c, grid, g)
    mu = torch.empty((c["n"], c["nsave"]), dtype=torch.float64, device=DEV)
    for s in range(c["nsave"]):
        b = _interpolate(table, [ps[s, k].double() for k in range(3)], grid, c["grid"])
        p = ps[s, 3:].double().t()
        mu[:, s] = ((p * b).sum(1) / (p.norm(dim=1) * b.norm(dim=1))).clamp(-1.0, 1.0)
    return mu


def _exact_dmumu(c, seed):
    mu = _exact_mu(c, seed)
    lags = [int(v) for v in _lags(c)]
    edges = torch.as_tensor(_edges(c), device=DEV)
    nl, nb, n = len(lags), c["bins"], c["n"]
    sd = torch.zeros((nl, nb), dtype=torch.float64, device=DEV)
    sd2 = torch.zeros_like(sd)
    per = torch.zeros((n, nl), dtype=torch.float64, device=DEV)
    cnt = torch.zeros((n, nl), dtype=torch.float64, device=DEV)
    starts = 1 if c["mode"] == "injection" else c["nsave"]
    chunk = max(1, (1 << 26) // c["nsave"])
    for i in range(0, n, chunk):
        m = mu[i:i + chunk].double()
        v = m[:, :starts].abs() if c.get("abs", True) else m[:, :starts]
        b = torch.bucketize(v, edges, right=True) - 1
        b = torch.where(v == edges[-1], nb - 1, b)
        b = torch.where((v >= edges[0]) & (v <= edges[-1]), b, nb).contiguous()
        for l, lag in enumerate(lags):
            k = min(starts, c["nsave"] - lag)
            if k <= 0:
                continue
            d = m[:, lag:lag + k] - m[:, :k]
            ok = torch.isfinite(d)
            d = torch.where(ok, d, 0.0)
            z = torch.zeros((m.shape[0], nb + 1), dtype=torch.float64, device=DEV)
            sd[l] += z.scatter_add_(1, b[:, :k], d).sum(0)[:nb]
            d = d * d
            z.zero_()
            sd2[l] += z.scatter_add_(1, b[:, :k], d).sum(0)[:nb]
            per[i:i + chunk, l] = d.sum(1)
            cnt[i:i + chunk, l] = ok.sum(1)
    used = cnt > 0
    value = torch.where(used, per / cnt.clamp_min(1.0), 0.0)
    num = used.sum(0).double()
    mean = value.sum(0) / num.clamp_min(1.0)
    m2 = torch.where(used, (value - mean) ** 2, 0.0).sum(0)
    return {"particle_counts": None, "particle_means": mean, "particle_m2s": m2, "pair_sum_squares": per.sum(0),
            "pair_counts": None, "dmumu_counts": None, "dmumu_sum_delta": sd, "dmumu_sum_delta2": sd2}


def _exact_dpp(c, seed):
    mom = _momenta(c, _gen(seed))
    lags = [int(v) for v in _lags(c)]
    p0 = _p(10.0)
    out = {k: torch.zeros(len(lags), dtype=torch.float64, device=DEV) for k in ("sum_delta_p", "sum_delta_p2")}
    mag = torch.empty((c["nsave"], c["n"]), dtype=torch.float64, device=DEV)
    for s in range(0, c["nsave"], 256):
        mag[s:s + 256] = (mom[s:s + 256].double() / p0).norm(dim=1)
    for l, lag in enumerate(lags):
        for i in range(0, c["nsave"] - lag, 1024):
            k = min(1024, c["nsave"] - lag - i)
            d = mag[i + lag:i + lag + k] - mag[i:i + k]
            d = torch.where(torch.isfinite(d), d, 0.0)
            out["sum_delta_p"][l] += d.sum()
            out["sum_delta_p2"][l] += (d * d).sum()
    at = np.linspace(0, c["nsave"] - 1, c["snaps"]).round().astype(np.int64)
    q = mag[torch.as_tensor(at, device=DEV)].t() * (p0 / (MP * C))
    energy = q * q / (torch.sqrt(1.0 + q * q) + 1.0) * (MP * C * C / (1e9 * QE))
    return {"energy": energy, "hist": None, "counts": None, "sum_delta_p": out["sum_delta_p"] * p0,
            "sum_delta_p2": out["sum_delta_p2"] * p0 * p0, "sum_delta_p_norm": out["sum_delta_p"],
            "sum_delta_p_norm2": out["sum_delta_p2"]}


def exact(case, seed):
    c = dict(case)
    if c["kind"] in ("push32", "host") and not _follows(c, c["energy"], c.get("steps") or c["nsteps"] - 1):
        return None
    if c["kind"] in ("push32", "push64", "host", "batch"):
        return _exact_push(c, seed)
    if c["kind"] in ("dmumu", "dmumu_ps"):
        return _exact_dmumu(c, seed)
    return _exact_dpp(c, seed)
