"""Performance cases: what users of the particle-move engine have it do, from the smallest calls to
the largest, through the public entry points (the Engine, the C ABI behind it, the training step).

Each case is a plain dict; `kind` names the way a program drives the library:

  host       records in the caller's (page-locked) host buffer, one forcing interval per call: the
             reference's own calling pattern. The records move on from pass to pass.
  day        a small release run resident for several hourly intervals, then read back.
  realistic  hourly production on a large ROMS-shaped grid: emission from point sources, the random
             walk, concentration and compaction each hour.
  batch      drift scenarios (leeway, wind, Stokes drift) as one CUDA graph over several hours.
  learned    the learned form: a surrogate displacement per interval, with or without the plain
             random walk on top.
  train      one training step of the surrogate (forward, backward, Adam).
  launcher   the reference's GPU launcher signature on the caller's device buffers.

`exact` gives, in 64 bits and with torch alone, what `run` returns.
"""
import ctypes
import math

import numpy as np
import torch

from wacommplusplus_b200 import _native
from wacommplusplus_b200 import surrogate
from wacommplusplus_b200 import synthetic
from wacommplusplus_b200 import surrogate_train
from wacommplusplus_b200.engine import Engine
from wacommplusplus_b200.types import PARTICLE_DTYPE, default_config, make_sources

HOUR = 3600.0
T_START = synthetic.EPOCH_2021_07_01
FLOAT_FIELDS = ("k", "j", "i", "health", "age")


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # The smallest call: a search-and-rescue sized release on a small nest, default options
        # (FP32 step, the reference's random keys), records in host memory, an hour per call.
        {"name": "host_1k_default", "kind": "host", "n": 1021, "eta": 32, "xi": 32, "levels": 10,
         "arithmetic": "fp32", "storage": "fp32", "rng": "reference", "walk": True,
         "backward": False, "dti": 30.0},
        # The parity-sized analytic case, tracked backward in the FP64 mode (source attribution).
        {"name": "host_16k_fp64_backward", "kind": "host", "n": 16384, "eta": 128, "xi": 128,
         "levels": 10, "arithmetic": "reference", "storage": "fp32", "rng": "reference",
         "walk": False, "backward": True, "dti": 30.0},
        # A day of a small release kept on the device, default options, read back at the end.
        {"name": "day_20k_default", "kind": "day", "n": 20011, "eta": 128, "xi": 128, "levels": 10,
         "hours": 12, "rng": "reference", "dti": 30.0},
        # An ordinary production population under the default options.
        {"name": "host_1m_default", "kind": "host", "n": 1048573, "eta": 128, "xi": 128,
         "levels": 10, "arithmetic": "fp32", "storage": "fp32", "rng": "reference", "walk": True,
         "backward": False, "dti": 30.0},
        # The FP64 mode with the reference's random walk at production size.
        {"name": "host_500k_fp64_walk", "kind": "host", "n": 500009, "eta": 131, "xi": 113,
         "levels": 10, "arithmetic": "reference", "storage": "fp32", "rng": "reference",
         "walk": True, "backward": False, "dti": 30.0},
        # Half-precision forcing storage, deterministic tracking.
        {"name": "host_4m_fp16", "kind": "host", "n": 4000037, "eta": 128, "xi": 128, "levels": 10,
         "arithmetic": "fp32", "storage": "fp16", "rng": "philox", "walk": False,
         "backward": False, "dti": 30.0},
        # The precision workload end to end: 16 Mi records from and to pinned memory, FP32.
        {"name": "host_16m", "kind": "host", "n": 1 << 24, "eta": 128, "xi": 128, "levels": 10,
         "arithmetic": "fp32", "storage": "fp32", "rng": "philox", "walk": False,
         "backward": False, "dti": 30.0},
        # Two hours of production on a ROMS-shaped grid with land.
        {"name": "realistic_2m", "kind": "realistic", "n": 2000000, "eta": 640, "xi": 768,
         "levels": 24, "sources": 64, "dti": 15.0},
        # Drift scenarios with wind and Stokes drift, six hours as one graph.
        {"name": "batch_400k", "kind": "batch", "n": 400000, "eta": 128, "xi": 128, "levels": 10,
         "hours": 6, "scenarios": 32, "dti": 30.0},
        # The learned form on a non-uniform flow: the surrogate with the random walk on top.
        {"name": "learned_1m_walk", "kind": "learned", "n": 1000003, "eta": 128, "xi": 128,
         "levels": 10, "hours": 2, "walk": True, "dti": 30.0},
        # One training step of the surrogate at the trainer's default batch.
        {"name": "train_16k", "kind": "train", "batch": 16384},
        # The reference's GPU launcher on device buffers of the caller.
        {"name": "launcher_500k", "kind": "launcher", "n": 524287, "eta": 128, "xi": 128,
         "levels": 10, "walk": False, "dti": 30.0},
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["host", "host", "host", "day", "realistic", "batch", "learned", "train",
                       "launcher"])
    case = {"kind": kind}
    if kind == "train":
        case["batch"] = _log_uniform(rng, 500, 65536)
        return case
    case["eta"], case["xi"] = rng.randint(24, 200), rng.randint(24, 200)
    case["levels"] = rng.randint(4, 20)
    case["dti"] = rng.choice([20.0, 30.0, 36.0, 60.0])
    if kind == "host":
        case["arithmetic"] = rng.choice(["fp32", "fp32", "fp32", "reference"])
        full = case["arithmetic"] == "reference"
        case["storage"] = "fp32" if full else rng.choice(["fp32", "fp32", "fp16", "bf16"])
        case["rng"] = rng.choice(["reference", "philox"])
        case["walk"] = rng.random() < 0.5
        case["backward"] = not case["walk"] and rng.random() < 0.4
        heavy = full or (case["walk"] and case["rng"] == "reference")
        case["n"] = _log_uniform(rng, 500, 600000 if full else 1500000 if heavy else 8000000)
    elif kind == "day":
        case["n"] = _log_uniform(rng, 500, 60000)
        case["hours"] = rng.randint(3, 12)
        case["rng"] = rng.choice(["reference", "philox"])
    elif kind == "realistic":
        case["eta"], case["xi"] = rng.randint(96, 640), rng.randint(96, 640)
        case["levels"], case["sources"] = rng.randint(8, 24), rng.randint(4, 64)
        case["n"] = _log_uniform(rng, 20000, 1500000)
        case["dti"] = 15.0
    elif kind == "batch":
        case["n"], case["hours"] = _log_uniform(rng, 20000, 400000), rng.randint(2, 6)
        case["scenarios"] = rng.randint(4, 64)
    elif kind == "learned":
        case["n"], case["hours"] = _log_uniform(rng, 20000, 1000000), 2
        case["walk"] = rng.random() < 0.5
    else:
        case["n"], case["walk"] = _log_uniform(rng, 2000, 500000), rng.random() < 0.3
    return case


# ------------------------------------------------------------------ inputs

def _seeded(seed):
    return np.random.default_rng(int(seed) % (1 << 31))


def _window(case, seed, frames):
    """A basin without land: a closed, slowly turning gyre field (rms 0.25 m/s), currents that
    decay with depth, a weak vertical velocity, log-normal diffusivity, a gently varying bottom.
    Records are hourly."""
    rng = _seeded(seed)
    eta, xi, levels = case["eta"], case["xi"], case["levels"]
    lon, lat, lon_rad, lat_rad = synthetic.rectilinear_grid(
        eta, xi, 14.0, 14.0 + 0.0016 * (xi - 1), 40.7, 40.7 + 0.0016 * (eta - 1))
    sw = np.arange(-levels, 1) / levels
    y, x = np.linspace(0, 1, eta)[:, None], np.linspace(0, 1, xi)[None, :]
    modes = [(m, n, rng.standard_normal(), rng.uniform(0, 2 * np.pi), rng.uniform(-0.4, 0.4))
             for m in (1, 2, 3) for n in (1, 2, 3)]
    u, v = np.zeros((frames, eta, xi)), np.zeros((frames, eta, xi))
    for m, n, amp, phase, omega in modes:
        scale = amp / math.hypot(m, n)
        for t in range(frames):
            a = scale * math.cos(phase + omega * t)
            u[t] -= a * n * np.sin(m * np.pi * x) * np.cos(n * np.pi * y)
            v[t] += a * m * np.cos(m * np.pi * x) * np.sin(n * np.pi * y)
    norm = 0.25 / math.sqrt(0.5 * (np.mean(u * u) + np.mean(v * v)))
    decay = 1.0 + 0.6 * 0.5 * (sw[1:] + sw[:-1])
    bell = np.sin(np.pi * sw)[None, :, None, None] * 2.0e-4
    swell = np.cos(3 * np.pi * x) * np.cos(2 * np.pi * y)
    hours = np.arange(frames)[:, None, None]
    noise = rng.standard_normal((frames, levels + 1, eta, xi), dtype=np.float32)
    return synthetic.Window(
        times=T_START + HOUR * np.arange(frames, dtype=np.float64), mask=np.ones((eta, xi)),
        lon=lon, lat=lat, lonRad=lon_rad, latRad=lat_rad, h=50.0 + 8.0 * swell, sWValues=sw,
        depthIntervals=np.ascontiguousarray(np.diff(sw)),
        zeta=(0.2 * np.sin(hours / 2.0 + 2 * np.pi * x[None])).astype(np.float32) + np.zeros(
            (frames, eta, xi), np.float32),
        u=(norm * decay[None, :, None, None] * u[:, None]).astype(np.float32),
        v=(norm * decay[None, :, None, None] * v[:, None]).astype(np.float32),
        w=(bell * swell[None, None] * np.cos(hours[..., None] / 3.0)).astype(np.float32),
        akt=(1.0e-4 * np.exp(noise)).astype(np.float32))


def _records(case, seed, time=T_START, late=0.0):
    """n records spread over the basin in its upper half, in page-locked memory, as a uint8
    tensor and its record view; `late`: the share released during the first hour."""
    n = case["n"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 7 + 3)
    draw_ = torch.rand((4, n), generator=gen, device="cuda", dtype=torch.float64)
    cols = torch.zeros((n, 8), device="cuda", dtype=torch.float64)
    cols[:, 0] = torch.arange(n, device="cuda", dtype=torch.int64).view(torch.float64)
    cols[:, 1] = -draw_[0] * 0.4 * case["levels"]
    cols[:, 2] = 0.5 + draw_[1] * (case["eta"] - 2)
    cols[:, 3] = 0.5 + draw_[2] * (case["xi"] - 2)
    cols[:, 4] = 1.0
    cols[:, 6] = time
    if late:
        cols[:, 6] += torch.where(draw_[3] < late, draw_[3] / late * HOUR, 0.0)
    pinned = torch.empty((n, 64), dtype=torch.uint8, pin_memory=True)
    pinned.copy_(cols.view(torch.uint8))
    return pinned, pinned.numpy().reshape(-1).view(PARTICLE_DTYPE)


def _config(case, **more):
    """A conservative tracer (a decay time of a month) under the reference's default closures."""
    return default_config(random=bool(case.get("walk", True)), dti=case["dti"],
                          tau0=30 * 86400.0, survprob=1e-30, **more)


def _counts(case, times):
    """A page-locked buffer for the concentration grid."""
    return torch.empty((times, case["levels"], case["eta"], case["xi"]), dtype=torch.int32,
                       pin_memory=True)


def _columns(pinned):
    """The moved records of a page-locked buffer, field by field."""
    values = pinned.view(torch.float64)
    out = {name: values[:, c] for name, c in zip(FLOAT_FIELDS, (1, 2, 3, 4, 5))}
    out["side"] = pinned[:, 58].view(torch.int8)
    return out


def prepare(case, seed):
    state = {"case": dict(case), "t": 0}
    kind = case["kind"]
    if kind == "train":
        state.update(_training(case, seed))
        return state
    if kind == "realistic":
        state.update(_realistic(case, seed))
        return state
    if kind == "launcher":
        state.update(_launcher(case, seed))
        return state
    hours = case.get("hours", 3)
    win = _window(case, seed, hours + 1)
    state["pinned"], state["records"] = _records(case, seed, late=0.25 if kind == "day" else 0.0)
    if kind == "host":
        first = hours if case["backward"] else 0
        state["records"]["time"] = win.times[first]
        state["t"], state["first"], state["last"] = first, first, 0 if case["backward"] else hours
        engine = Engine(0, arithmetic=case["arithmetic"], storage=case["storage"],
                        rng=case["rng"])
        engine.set_config(_config(case, trackingDirection=-1 if case["backward"] else 1))
        engine.load_window(win)
    elif kind == "day":
        engine = Engine(0, rng=case["rng"])
        engine.set_config(_config(case))
        engine.load_window(win)
        engine.concentration_reset(hours + 1)
        state["counts"] = _counts(case, hours + 1)
        state["back"] = torch.empty_like(state["pinned"], pin_memory=True)
    elif kind == "batch":
        engine = _batch(case, seed, win, state)
    else:
        engine = Engine(0, storage="fp16", rng="philox")
        engine.set_surrogate()
        engine.set_options(surrogate=True)
        engine.set_config(_config(case))
        engine.load_window(win)
        state["back"] = torch.empty_like(state["pinned"], pin_memory=True)
    state["engine"], state["hours"] = engine, hours
    return state


def _scenario_records(case, seed, records):
    """Scenario attributes of a batch: a source, a release window and a leeway object each."""
    rng = _seeded(seed + 17)
    count = case["scenarios"]
    cuts = np.sort(rng.integers(0, case["n"], count - 1))
    for a, b in zip(np.r_[0, cuts], np.r_[cuts, case["n"]]):
        r, m = records[a:b], b - a
        r["j"] = rng.uniform(6, case["eta"] - 7) + 0.25 * rng.standard_normal(m)
        r["i"] = rng.uniform(6, case["xi"] - 7) + 0.25 * rng.standard_normal(m)
        r["k"] = -0.1 * case["levels"] * rng.uniform(0, 1, m)
        start = rng.uniform(0, 0.5 * case["hours"]) * HOUR
        r["time"] = T_START + start + (np.arange(m) + 0.5) * (HOUR / max(m, 1))
        r["driftObjectType"] = rng.integers(1, 23)
        r["driftSide"] = rng.choice(np.array([-1, 1], np.int8), m)


def _environment(case, seed, frames):
    """Smooth wind (rms 8 m/s) and Stokes drift (rms 0.1 m/s) at the rho nodes, hourly."""
    shape = (case["eta"], case["xi"])
    wu, wv = synthetic.vector_series(shape, frames, 8.0, int(seed) % 100003, 10.0)
    su, sv = synthetic.vector_series(shape, frames, 0.1, int(seed) % 100003 + 1, 6.0, 8.0)
    return wu, wv, su, sv


def _batch(case, seed, win, state):
    _scenario_records(case, seed, state["records"])
    win.windU10, win.windV10, win.stokesU, win.stokesV = _environment(case, seed, win.T)
    engine = Engine(0, rng="philox")
    engine.set_config(_config(case, driftModel=1, hasWind=True))
    engine.load_window(win)
    engine.concentration_reset(win.T)
    engine.set_particles(state["records"])
    engine.graph_capture(0, case["hours"])
    state["counts"] = _counts(case, win.T)
    state["back"] = torch.empty_like(state["pinned"], pin_memory=True)
    return engine


def _realistic(case, seed):
    forcing = synthetic.RealisticForcing(eta=case["eta"], xi=case["xi"], s_rho=case["levels"],
                                         n_frames=3, seed=int(seed) % 100003)
    win = forcing.window_of(range(3), [forcing.frame_device(t) for t in range(3)])
    per_hour = case["n"] / case["sources"]
    day = win.times[0] / 86400.0
    rows = [(k, j, i, day, day + 1.0 / 24, per_hour, "uniform_rate")
            for k, j, i in forcing.sources(case["sources"], seed=int(seed) % 100003 + 1)]
    engine = Engine(0, rng="philox")
    engine.set_config(_config(case))
    engine.load_window(win)
    engine.concentration_reset(3)
    return {"engine": engine, "sources": make_sources(rows), "times": win.times, "hours": 2,
            "counts": _counts(case, 3)}


def _training(case, seed):
    """Rows as the trainer meets them: stencil features, offsets, gates and residuals."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) + 11)
    rows = case["batch"]
    base = torch.randn((rows, 12), generator=gen, device="cuda")
    stencil = 0.3 * (base @ torch.randn((12, 384), generator=gen, device="cuda")) / math.sqrt(12)
    stencil += 0.05 * torch.randn((rows, 384), generator=gen, device="cuda")
    particle = torch.rand((rows, 4), generator=gen, device="cuda")
    gate = torch.rand(rows, generator=gen, device="cuda")
    residual = base[:, :3] * 0.5 + 0.1 * torch.randn((rows, 3), generator=gen, device="cuda")
    trainer = surrogate_train.KernelTrainer(torch, surrogate.random_weights(int(seed) % 100003),
                                            rows)
    return {"trainer": trainer, "batch": (stencil, particle, gate, residual)}


def _launcher(case, seed):
    win = _window(case, seed, 2)
    pinned, _ = _records(case, seed)
    cfg = default_config(random=case["walk"], dti=case["dti"], tau0=30 * 86400.0, survprob=1e-30)
    up = lambda a, kind: torch.as_tensor(np.ascontiguousarray(a, kind)).cuda()  # noqa: E731
    f64 = [up(a, np.float64) for a in (win.times, win.mask, win.lonRad, win.latRad,
                                       win.depthIntervals, win.h)]
    f32 = [up(a, np.float32) for a in (win.zeta, win.u, win.v, win.w, win.akt)]
    records = pinned.cuda()
    config = torch.frombuffer(bytearray(bytes(cfg)), dtype=torch.uint8).cuda()
    args = [config.data_ptr(), records.data_ptr(), 0, 2, win.sW, win.sRho, win.eta, win.xi]
    args += [a.data_ptr() for a in f64 + f32] + [None] * 4 + [case["n"], 1, 1]
    return {"args": args, "device": records, "keep": (config, f64, f32),
            "launch": _native.lib().wacomm_b200_cuda_move_particle}


# ------------------------------------------------------------------ one pass

def _read_back(engine, pinned):
    """The resident records into a page-locked buffer through the C ABI."""
    engine._check(engine._lib.wacomm_b200_get_particles(
        engine._ctx, ctypes.c_void_p(pinned.data_ptr()), len(pinned)))
    return _columns(pinned)


def _read_counts(engine, counts):
    """The concentration grid into a page-locked buffer (int32 holding the uint32 counts)."""
    engine._check(engine._lib.wacomm_b200_concentration_get(
        engine._ctx, ctypes.c_void_p(counts.data_ptr()), counts.numel()))
    return counts


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "host":
        engine, t = state["engine"], state["t"]
        engine.move_interval_host_ptr(t, state["pinned"].data_ptr(), case["n"])
        t += -1 if case["backward"] else 1
        state["t"] = state["first"] if t == state["last"] else t
        return _columns(state["pinned"])
    if kind == "day":
        engine = state["engine"]
        engine.set_particles(state["records"])
        engine.concentration_reset(state["hours"] + 1)
        for t in range(state["hours"]):
            engine.move_interval(t)
        out = _read_back(engine, state["back"])
        out["concentration"] = _read_counts(engine, state["counts"])
        return out
    if kind == "realistic":
        engine, times = state["engine"], state["times"]
        engine.set_particles(np.zeros(0, PARTICLE_DTYPE))
        engine.concentration_reset(3)
        emitted = engine.emit(state["sources"], times[0], times[1])
        for t in range(state["hours"]):
            engine.move_interval(t)
            engine.remove_dead()
        return {"concentration": _read_counts(engine, state["counts"]), "emitted": emitted,
                "left": engine.count()}
    if kind == "batch":
        engine = state["engine"]
        engine.set_particles(state["records"])
        engine.concentration_reset(case["hours"] + 1)
        engine.graph_launch()
        out = _read_back(engine, state["back"])
        out["concentration"] = _read_counts(engine, state["counts"])
        return out
    if kind == "learned":
        engine = state["engine"]
        engine.set_particles(state["records"])
        for t in range(state["hours"]):
            engine.move_interval(t)
        return _read_back(engine, state["back"])
    if kind == "train":
        trainer = state["trainer"]
        loss = trainer.run(*state["batch"], lr=1e-3)
        return {"loss": loss, "grads": trainer.grads, "params": trainer.params, "m": trainer.m,
                "v": trainer.v}
    status = state["launch"](*state["args"], torch.cuda.current_stream().cuda_stream)
    if status != 0:
        raise RuntimeError(f"the launcher failed ({status})")
    return _columns(state["device"])


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Bytes: records read and written once, every forcing record used read once, the
    concentration grid written once. Operations: per substep, two velocity interpolations (one
    for the learned form's random walk), the diffusivity, the column heights, the landing."""
    if case["kind"] == "train":
        rows = case["batch"]
        weights = surrogate.N_PARAMETERS
        return {"bytes": 4.0 * (rows * (388 + 1 + 3) + 7 * weights),
                "flops": 2.0 * rows * (2 * 388 * 256 + 6 * 256 * 256)}
    plane = case["eta"] * case["xi"]
    record = 4.0 * plane * (1 + 2 * case["levels"] + 2 * (case["levels"] + 1))
    hours = case.get("hours", 2 if case["kind"] == "realistic" else 1)
    walk = case.get("walk", True)
    per_step = 170.0 + (90.0 if walk else 0.0) + (110.0 if case["kind"] == "batch" else 0.0)
    steps = case["n"] * math.ceil(HOUR / case["dti"]) * hours
    move = 128.0 * case["n"] + record * (hours + 1)
    if case["kind"] == "realistic":
        steps *= 0.75  # released evenly over the first of the two hours
        return {"bytes": move + 4.0 * 3 * plane * case["levels"], "flops": per_step * steps}
    if case["kind"] in ("day", "batch"):
        move += 4.0 * (hours + 1) * plane * case["levels"]
    if case["kind"] == "learned":
        mlp = 2.0 * (384 * 256 * (case["eta"] - 1) * (case["xi"] - 1) * case["levels"] +
                     case["n"] * (4 * 256 + 2 * 256 * 256 + 3 * 256))
        return {"bytes": move, "flops": hours * mlp + (110.0 * steps if walk else 0.0)}
    return {"bytes": move, "flops": per_step * steps}


# ------------------------------------------------------------------ the same in 64 bits

MASK32 = 0xFFFFFFFF


def _signed(value):
    return value - (1 << 64) if value >= 1 << 63 else value


def _shift(x, bits):
    return (x >> bits) & ((1 << (64 - bits)) - 1)


def _mix(x):
    x = x + _signed(0x9E3779B97F4A7C15)
    x = (x ^ _shift(x, 30)) * _signed(0xBF58476D1CE4E5B9)
    x = (x ^ _shift(x, 27)) * _signed(0x94D049BB133111EB)
    return x ^ _shift(x, 31)


def _uniform(key):
    return _shift(key, 11).double() * 2.0 ** -53


def _ordered_normals(prefix, substep):
    """Three normals of the ordered SplitMix64 keys."""
    key = _mix(prefix ^ substep)
    out = []
    for c in range(3):
        u1 = _uniform(_mix(key ^ (2 * c))).clamp(min=2.2250738585072014e-308)
        u2 = _uniform(_mix(key ^ (2 * c + 1)))
        out.append(torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(2 * math.pi * u2))
    return out


def _philox_normals(key, interval, elapsed):
    """Three normals of the Philox4x32-10 stream of (key, interval, elapsed time)."""
    bits = elapsed.view(torch.int64)
    x, y = bits & MASK32, _shift(bits, 32)
    z = torch.full_like(x, interval & MASK32)
    w = torch.full_like(x, (interval >> 32) & MASK32)
    k0, k1 = key & MASK32, _shift(key, 32)
    for _ in range(10):
        p0, p1 = x * 0xD2511F53, z * 0xCD9E8D57
        x, y, z, w = (_shift(p1, 32) ^ y ^ k0, p1 & MASK32, _shift(p0, 32) ^ w ^ k1, p0 & MASK32)
        k0, k1 = (k0 + 0x9E3779B9) & MASK32, (k1 + 0xBB67AE85) & MASK32
    u0, u1 = (x.double() + 1) * 2.0 ** -32, y.double() * 2.0 ** -32
    u2, u3 = (z.double() + 1) * 2.0 ** -32, w.double() * 2.0 ** -32
    r0, r2 = torch.sqrt(-2 * torch.log(u0)), torch.sqrt(-2 * torch.log(u2))
    a0, a2 = (2 * u1 - 1) * math.pi, (2 * u3 - 1) * math.pi
    return [r0 * torch.cos(a0), r0 * torch.sin(a0), r2 * torch.cos(a2)]


# Leeway coefficients of the catalogue's objects: downwind slope and offset, then the crosswind
# slope and offset to the right and to the left of the wind.
LEEWAY = [
    (0, 0, 0, 0, 0, 0), (.0096, 0, .0054, 0, -.0054, 0), (.0339, 0, .0149, 0, -.0149, 0),
    (.0121, 0, .0092, 0, -.0092, 0), (.0247, 0, .0276, 0, -.0276, 0),
    (.0125, .0396, .0019, .0114, -.0019, -.0114), (.0048, 0, .0015, 0, -.0015, 0),
    (.0171, .0112, .0136, -.033, -.0013, -.0265), (.01117, .102, .0004, .039, -.0004, -.039),
    (.0352, -.025, .0062, -.03, -.0045, -.002), (.0088, 0, .0018, 0, -.0018, 0),
    (.0116, .1112, .0041, 0, -.0041, 0), (.0193, 0, .0051, 0, -.0051, 0),
    (.0315, 0, .0129, 0, -.0129, 0), (.0165, 0, .0039, 0, -.0039, 0),
    (.0654, 0, .0219, 0, -.0219, 0), (.0187, 0, .0209, 0, -.0209, 0),
    (.045, 0, .0495, 0, -.0282, 0), (.0197, 0, .0036, 0, -.0036, 0),
    (.0075, .0266, .0048, .0288, -.0045, -.0146), (.0107, .0447, .0041, .0115, -.0041, -.0115),
    (.0156, .083, .00078, .027, -.00078, -.027), (.0275, 0, .005, 0, -.005, 0)]


class _Basin:
    """The forcing of one interval and the particle step on it, in 64 bits."""

    def __init__(self, win, t, direction, environment):
        up = lambda a: torch.as_tensor(np.asarray(a), device="cuda").double()  # noqa: E731
        self.eta, self.xi, self.levels = win.eta, win.xi, win.sRho
        self.start, self.end = float(win.times[t]), float(win.times[t + direction])
        pair = (t, t + direction)
        flat = lambda name: [up(getattr(win, name)[s]).reshape(-1) for s in pair]  # noqa: E731
        self.rho = torch.stack(flat("u") + flat("v"), 1)
        self.wet = torch.stack(flat("w") + flat("akt"), 1)
        self.top = torch.stack([up(win.h).reshape(-1)] + flat("zeta"), 1)
        self.env = None
        if environment is not None:
            self.env = torch.stack([up(a[s]).reshape(-1) for a in environment for s in pair], 1)
        self.depth = up(win.depthIntervals)
        x, y = surrogate_metric(win.lonRad, win.latRad)
        self.metric = torch.stack([up(x).reshape(-1), up(y).reshape(-1)], 1)

    def corners(self, table, cell, jf, if_, plane=0):
        at = cell + plane
        return (table[at] * ((1 - if_) * (1 - jf))[:, None] +
                table[at + self.xi] * ((1 - if_) * jf)[:, None] +
                table[at + self.xi + 1] * (if_ * jf)[:, None] +
                table[at + 1] * (if_ * (1 - jf))[:, None])

    def locate(self, j, i):
        jc, ic = torch.floor(j), torch.floor(i)
        ok = (jc >= 0) & (ic >= 0) & (jc + 1 < self.eta) & (ic + 1 < self.xi)
        jc, ic = jc.clamp(0, self.eta - 2), ic.clamp(0, self.xi - 2)
        return ok, jc.long() * self.xi + ic.long(), j - jc, i - ic

    def column(self, cell, jf, if_, a):
        top = self.corners(self.top, cell, jf, if_)
        return top[:, 0] + (1 - a) * top[:, 1] + a * top[:, 2]

    def vertical(self, k):
        kc = torch.ceil(k)
        return kc.clamp(-self.levels + 1, 0).long(), kc - k

    def velocity(self, level, kf, cell, jf, if_, a, drift):
        plane = self.eta * self.xi
        up = (level + self.levels) * plane
        h = self.corners(self.rho, cell, jf, if_, up - plane)
        u, v = (1 - a) * h[:, 0] + a * h[:, 1], (1 - a) * h[:, 2] + a * h[:, 3]
        w = (self.corners(self.wet, cell, jf, if_, up) * (1 - kf)[:, None] +
             self.corners(self.wet, cell, jf, if_, up - plane) * kf[:, None])
        if drift is not None:
            e = self.corners(self.env, cell, jf, if_)
            wu, wv, su, sv = ((1 - a) * e[:, 2 * c] + a * e[:, 2 * c + 1] for c in range(4))
            table, side = drift
            speed = torch.sqrt(wu * wu + wv * wv).clamp(min=1e-300)
            right = side == 1
            down = table[:, 0] * speed + table[:, 1]
            cross = torch.where(right, table[:, 2] * speed + table[:, 3],
                                table[:, 4] * speed + table[:, 5])
            u = u + (down * wu - cross * wv) / speed + su
            v = v + (down * wv + cross * wu) / speed + sv
        akt = lambda alpha: (1 - alpha) * w[:, 2] + alpha * w[:, 3]  # noqa: E731
        return u, v, (1 - a) * w[:, 0] + a * w[:, 1], akt


def surrogate_metric(lon, lat):
    """Cell sizes in metres along i and j: haversine along each axis."""
    lon, lat = np.asarray(lon, np.float64), np.asarray(lat, np.float64)
    x, y = np.ones(lon.shape), np.ones(lon.shape)
    d = np.sin(0.5 * (lat[1:, :-1] - lat[:-1, :-1])) ** 2
    y[:-1, :-1] = 2 * np.arctan2(np.sqrt(d), np.sqrt(1 - d)) * 6371000.0
    d = (np.sin(0.5 * (lon[:-1, 1:] - lon[:-1, :-1])) ** 2 * np.cos(lat[:-1, 1:]) *
         np.cos(lat[:-1, :-1]))
    x[:-1, :-1] = 2 * np.arctan2(np.sqrt(d), np.sqrt(1 - d)) * 6371000.0
    return x, y


def _reflect(x, top):
    x = x.abs()
    x = torch.where(x >= top, 2 * top - x, x)
    return torch.where(x >= top, torch.full_like(x, math.nextafter(top, 0.0)), x)


def _bounce(k, dead, lower):
    """The vertical closures: held at the surface, removed at the bottom."""
    return k.clamp(max=0.0), dead | (k < lower)


def _interval(basin, p, case, cfg, direction, drift=None, rates=None):
    """One interval of every record in p (k, j, i, age, time, id, dead), every substep; with
    `rates` the deterministic displacement is those constant velocities (the learned form)."""
    length = abs(basin.end - basin.start)
    lower = float(-basin.levels + 1)
    key = _signed(0) + int(round(min(basin.start, basin.end)))
    seed = _mix(torch.tensor([_signed(cfg["seed"])], device="cuda"))
    prefix = _mix(_mix(seed ^ p["id"]) ^ key)
    stream = p["id"] ^ seed
    k, j, i, age, dead = p["k"], p["j"], p["i"], p["age"], p["dead"]
    elapsed = torch.zeros_like(k)
    if direction > 0:
        elapsed = (p["time"] - basin.start).clamp(0.0, length)
    dti = case["dti"]
    while True:
        ok, cell, jf, if_ = basin.locate(j, i)
        dead = dead | (~ok & (elapsed < length))
        live = (elapsed < length) & ~dead
        if not bool(live.any()):
            break
        dt = torch.minimum(torch.full_like(k, dti), length - elapsed)
        dt = torch.where(live, dt, torch.ones_like(dt))
        a, a0 = (elapsed + 0.5 * dt) / length, elapsed / length
        level, kf = basin.vertical(k)
        height = basin.column(cell, jf, if_, a)
        size = basin.metric[cell]
        xd, yd = size[:, 0], size[:, 1]
        zd = height * basin.depth[level + basin.levels - 1]
        u, v, w, akt = basin.velocity(level, kf, cell, jf, if_, a0, drift)
        rx = ry = rz = 0.0
        if cfg["walk"]:
            n = (_philox_normals(stream, key, elapsed) if cfg["rng"] == "philox"
                 else _ordered_normals(prefix, torch.floor(elapsed / dti).long()))
            sigma = 3.46 * (1 - k / lower) * torch.sqrt(dt / dti)
            rx, ry, rz = sigma * n[0], sigma * n[1], sigma * n[2] * akt(a)
        if rates is not None:
            dx, dy, dz = rates[0] * dt, rates[1] * dt, rates[2] * dt
        else:
            half = torch.maximum(torch.minimum(direction * w * 0.5 * dt, zd), -zd)
            km = (k + half / zd).clamp(lower, 0.0)
            okm, cm, jm, im = basin.locate(j + direction * v * 0.5 * dt / yd,
                                           i + direction * u * 0.5 * dt / xd)
            cm, jm, im = (torch.where(okm, m, s) for m, s in ((cm, cell), (jm, jf), (im, if_)))
            lm, fm = basin.vertical(torch.where(okm, km, k))
            um, vm, wm, _ = basin.velocity(lm, fm, cm, jm, im, a, drift)
            sm = basin.metric[cm]
            zm = torch.where(okm, basin.column(cm, jm, im, a) * basin.depth[lm + basin.levels - 1],
                             zd)
            dx = direction * um * dt * xd / sm[:, 0]
            dy = direction * vm * dt * yd / sm[:, 1]
            dz = direction * wm * dt * zd / zm
        dz = torch.maximum(torch.minimum(dz + rz, zd), -zd)
        jn, in_ = j + (dy + ry) / yd, i + (dx + rx) / xd
        kn, gone = _bounce(k + dz / zd, dead, lower)
        inside = basin.locate(jn, in_)[0]
        jn = torch.where(inside, jn, _reflect(jn, float(basin.eta - 1)))
        in_ = torch.where(inside, in_, _reflect(in_, float(basin.xi - 1)))
        k, j, i = (torch.where(live, n_, o) for n_, o in ((kn, k), (jn, j), (in_, i)))
        dead = torch.where(live, gone, dead)
        age = torch.where(live & ~gone, age + dt, age)
        elapsed = torch.where(live, elapsed + dt, elapsed)
    p.update(k=k, j=j, i=i, age=age, dead=dead)


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(0.7978845608028654 * (x + 0.044715 * x ** 3)))


def _learned_interval(basin, win, t, p, case, cfg, net):
    """One interval of the learned form: the network's correction to the displacement at the
    start point, in closed form without the random walk, as constant rates with it."""
    length = basin.end - basin.start
    eta, xi, levels = basin.eta, basin.xi, basin.levels
    a0 = ((p["time"] - basin.start) / length).clamp(0.0, 1.0)
    am, rest = 0.5 * (a0 + 1), (1 - a0) * length
    ok, cell, jf, if_ = basin.locate(p["j"], p["i"])
    jc, ic = cell // xi, cell % xi
    level, kf = basin.vertical(p["k"])
    four = torch.arange(4, device="cuda")
    rows = (jc[:, None] - 1 + four).clamp(0, eta - 1)
    cols = (ic[:, None] - 1 + four).clamp(0, xi - 1)
    planes = {n: (level[:, None] - 2 + four).clamp(-n + 1, 0) + n - 1 for n in (levels, levels + 1)}
    blocks = []
    for s in (t, t + 1):
        for name, count, scale in (("u", levels, 1.0), ("v", levels, 1.0),
                                   ("w", levels + 1, 1.0e3)):
            field = torch.as_tensor(getattr(win, name)[s], device="cuda").double().reshape(-1)
            at = (planes[count][:, :, None, None] * (eta * xi) + rows[:, None, :, None] * xi +
                  cols[:, None, None, :])
            blocks.append(field[at.reshape(len(jc), -1)] * scale)
    spread = sum(((b - b[:, 21:22]) ** 2).sum(1) for b in (blocks[0], blocks[1], blocks[3],
                                                           blocks[4]))
    gate = (torch.sqrt(spread / 256.0) / 0.01).clamp(max=1.0)
    x = torch.cat(blocks + [torch.stack([jf, if_, kf, a0], 1)], 1)
    for n in (1, 2, 3):
        x = _gelu(x @ net["w%d" % n].T + net["b%d" % n])
    y = (x @ net["w4"].T + net["b4"]) * gate[:, None]
    u, v, w, _ = basin.velocity(level, kf, cell, jf, if_, am, None)
    run_ = rest > 0
    safe = torch.where(run_, rest, torch.ones_like(rest))
    if cfg["walk"]:
        _interval(basin, p, case, cfg, 1, rates=(u + 100 * y[:, 0] / safe, v + 100 * y[:, 1] / safe,
                                                 w + y[:, 2] / safe))
        return
    size = basin.metric[cell]
    zd = basin.column(cell, jf, if_, am) * basin.depth[level + levels - 1]
    steps = torch.ceil(rest / case["dti"] - 1e-9).clamp(min=1)
    ends = []
    for x0, move, top in ((p["j"], (v * rest + 100 * y[:, 1]) / size[:, 1], float(eta - 1)),
                          (p["i"], (u * rest + 100 * y[:, 0]) / size[:, 0], float(xi - 1))):
        d, at = move / steps, x0.clone()
        for _ in range(int(steps.max())):
            nxt = at + d
            nxt = torch.where((nxt >= 0) & (nxt < top), nxt, _reflect(nxt, top))
            at = torch.where(_ < steps, nxt, at)
        ends.append(at)
    kn, gone = _bounce(p["k"] + (w * rest + y[:, 2]) / zd, p["dead"], float(-levels + 1))
    live = run_ & ok & ~p["dead"]
    p.update(j=torch.where(live, ends[0], p["j"]), i=torch.where(live, ends[1], p["i"]),
             k=torch.where(live, kn, p["k"]), age=torch.where(live, p["age"] + rest, p["age"]),
             dead=p["dead"] | (live & gone))


def _exact_training(case, seed):
    made = _training(case, seed)
    stencil, particle, gate, residual = (x.double() for x in made["batch"])
    net = {k: torch.as_tensor(v, device="cuda").double().requires_grad_(True)
           for k, v in surrogate.random_weights(int(seed) % 100003).items()}
    x = torch.cat([stencil, particle], 1)
    for n in (1, 2, 3):
        x = _gelu(x @ net["w%d" % n].T + net["b%d" % n])
    y = (x @ net["w4"].T + net["b4"]) * gate[:, None]
    loss = ((y - residual) ** 2).mean()
    loss.backward()
    names = [name for name, _ in surrogate.PARAMETERS]
    grads = torch.cat([net[n].grad.reshape(-1) for n in names])
    params = torch.cat([net[n].detach().reshape(-1) for n in names])
    # one Adam step divides each gradient by its own size: the sign alone is left, and the
    # weights move by the learning rate
    params = params - 1e-3 * grads / (grads.abs() + 1e-8)
    return {"loss": loss.detach().reshape(1), "grads": grads, "params": params, "m": 0.1 * grads,
            "v": 0.001 * grads * grads}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_training(case, seed)
    if kind == "realistic":
        return None  # whole numbers only
    hours = case.get("hours", 1 if kind == "launcher" else 3)
    win = _window(case, seed, hours + 1)
    backward = bool(case.get("backward"))
    first = hours if backward else 0
    pinned, records = _records(case, seed, late=0.25 if kind == "day" else 0.0)
    if kind == "host":
        records["time"] = win.times[first]
    environment = None
    if kind == "batch":
        _scenario_records(case, seed, records)
        environment = _environment(case, seed, hours + 1)
    cfg = {"walk": bool(case.get("walk", True)), "seed": 5489,
           "rng": case.get("rng", "reference" if kind == "launcher" else "philox")}
    net = None
    if kind == "learned":
        net = {k: torch.as_tensor(v, device="cuda").double()
               for k, v in surrogate.load_weights().items()}
    passes = range(hours) if kind in ("day", "batch", "learned") else [first]
    parts = []
    chunk = 1 << (18 if kind == "learned" else 21)
    up = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    for a in range(0, case["n"], chunk):
        r = records[a:a + chunk]
        p = {name: up(r[name]) for name in ("k", "j", "i", "age", "time")}
        p["id"] = up(r["id"].view(np.int64))
        p["dead"] = torch.zeros(len(r), dtype=torch.bool, device="cuda")
        drift = None
        if kind == "batch":
            table = torch.tensor(LEEWAY, device="cuda", dtype=torch.float64)
            drift = (table[up(r["driftObjectType"].astype(np.int64))], up(r["driftSide"]))
        for t in passes:
            basin = _Basin(win, t, -1 if backward else 1, environment)
            if kind == "learned":
                _learned_interval(basin, win, t, p, case, cfg, net)
            else:
                _interval(basin, p, case, cfg, -1 if backward else 1, drift)
        fresh = p["age"] == 0
        health = torch.where(p["dead"], -1.0, torch.where(fresh, 1.0,
                                                         torch.exp(-p["age"] / (30 * 86400.0))))
        parts.append({"k": p["k"], "j": p["j"], "i": p["i"], "health": health, "age": p["age"]})
    out = {name: torch.cat([q[name] for q in parts]) for name in FLOAT_FIELDS}
    out["side"] = None
    if kind in ("day", "batch"):
        out["concentration"] = None
    return out
