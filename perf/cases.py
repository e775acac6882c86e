"""The work that programs have this library do, as cases that can be timed and compared.

Every case goes through the public entry points of the host binding (hhs.py, the C ABI):

- hold:   one top-level HOLD step of a Plummer sphere (hold_step), the call that an
          integration repeats; mixed precision and FP64, with and without softening.
- batch:  one step of many independent clusters in one launch (Batch.step).
- level:  one level of the recursion through the reference-shaped calls (timesteps, split,
          drift, kick_slow, kick_sf both ways, update_system), as an integrator that keeps
          its own schedule makes them.
- scan, compact: the standalone exclusive scan and stream compaction of int32 flags.

Inputs are seeded; a pass starts from the same particle state each time (one device copy),
so that every pass of a case does the same work.
"""
import ctypes
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "parallel-hhs_b200"))

import hhs  # noqa: E402

PREC = {"mixed": hhs.PREC_MIXED, "fp64": hhs.PREC_FP64}
DT = 1.0 / 64  # the top-level step of every workload of the benchmark


def listed():
    return [
        # the smallest system that the tests and the smoke run step: all latency
        {"name": "hold_256_mixed", "kind": "hold", "n": 256, "prec": "mixed", "mass": 0,
         "eta": 0.03, "eps": 0.0},
        # plain FP64 HOLD, the benchmark's first configuration
        {"name": "hold_1024_fp64", "kind": "hold", "n": 1024, "prec": "fp64", "mass": 0,
         "eta": 0.03, "eps": 0.0},
        # an ordinary softened run of an odd size
        {"name": "hold_4099_mixed_soft", "kind": "hold", "n": 4099, "prec": "mixed", "mass": 2,
         "eta": 0.03, "eps": 1e-3},
        # the benchmark's headline configuration, and its accuracy reference in FP64
        {"name": "hold_16384_mixed", "kind": "hold", "n": 16384, "prec": "mixed", "mass": 0,
         "eta": 0.03, "eps": 0.0},
        {"name": "hold_16384_fp64", "kind": "hold", "n": 16384, "prec": "fp64", "mass": 0,
         "eta": 0.03, "eps": 0.0},
        # the deep hierarchy: Salpeter masses, the largest system here
        {"name": "hold_65536_salpeter", "kind": "hold", "n": 65536, "prec": "mixed", "mass": 1,
         "eta": 0.02, "eps": 0.0},
        # 512 clusters of 64 to 4096 particles in one launch
        {"name": "batch_512", "kind": "batch", "systems": 512, "lo": 64, "hi": 4096,
         "prec": "mixed", "eta": 0.03},
        # an integrator with a schedule of its own: one level, call by call
        {"name": "level_2051_fp64", "kind": "level", "n": 2051, "prec": "fp64", "mass": 0,
         "eta": 0.03},
        {"name": "level_16384_mixed", "kind": "level", "n": 16384, "prec": "mixed", "mass": 0,
         "eta": 0.03},
        # scan and compaction of flags: one level of a large system, and bulk data
        {"name": "scan_2p20", "kind": "scan", "n": 1 << 20, "p": 0.5},
        {"name": "scan_2p26", "kind": "scan", "n": 1 << 26, "p": 0.5},
        {"name": "compact_odd_2p24", "kind": "compact", "n": (1 << 24) + 4099, "p": 0.1},
    ]


def _log_size(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["hold", "hold", "hold", "hold", "batch", "level", "level", "scan",
                       "compact"])
    if kind == "hold":
        prec = rng.choice(["mixed", "mixed", "fp64"])
        return {"kind": "hold", "n": _log_size(rng, 64, 40000 if prec == "mixed" else 12000),
                "prec": prec, "mass": rng.choice([0, 1, 2]), "eta": rng.choice([0.02, 0.03]),
                "eps": rng.choice([0.0, 0.0, 1e-3])}
    if kind == "batch":
        return {"kind": "batch", "systems": _log_size(rng, 16, 512), "lo": 64,
                "hi": rng.choice([1024, 2048, 4096]), "prec": rng.choice(["mixed", "mixed", "fp64"]),
                "eta": rng.choice([0.02, 0.03])}
    if kind == "level":
        return {"kind": "level", "n": _log_size(rng, 256, 32768),
                "prec": rng.choice(["mixed", "fp64"]), "mass": rng.choice([0, 1, 2]),
                "eta": rng.choice([0.02, 0.03])}
    return {"kind": kind, "n": _log_size(rng, 1 << 16, 1 << 26), "p": rng.choice([0.01, 0.1, 0.5])}


# ------------------------------------------------------------------ device arrays
class _Array:
    """FP64 values of the library on the device, for torch.as_tensor (no copy)."""

    def __init__(self, ptr, count, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8",
                                         "data": (ptr, False), "version": 2}


def _address(p):
    return ctypes.cast(p, ctypes.c_void_p).value


def _block(system, first, last, n):
    """The fields first..last of a particle system as one array of rows (they are adjacent)."""
    a, b = _address(getattr(system.c, first)), _address(getattr(system.c, last))
    pitch = (_address(system.c.y) - _address(system.c.x)) // 8
    rows = (b - a) // 8 // pitch + 1
    flat = torch.as_tensor(_Array(a, rows * pitch, system), device="cuda")
    return flat.view(rows, pitch)[:, :n]


def _particles(parts, seeds, mass):
    """Plummer spheres one after another: the device system and what its passes start from."""
    whole = [hhs.plummer(int(n), int(s), mass) for n, s in zip(parts, seeds)]
    whole = {k: np.concatenate([p[k] for p in whole]) for k in whole[0]}
    n = len(whole["x"])
    system = hhs.ParticleSystem(n)
    system.upload(whole)
    torch.cuda.synchronize()
    state = {"system": system, "all": _block(system, "x", "ts", n),
             "pos": _block(system, "x", "z", n), "vel": _block(system, "vx", "vz", n),
             "mass": _block(system, "m", "m", n)[0]}
    state["start"] = state["all"].clone()
    return state


def _sizes(case):
    """Cluster sizes of a batch, log-uniform: the same for every seed of the particles."""
    rng = np.random.default_rng(case["systems"])
    return np.round(np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]),
                                       case["systems"]))).astype(np.int64)


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("scan", "compact"):
        n = case["n"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        flags = (torch.rand(n, device="cuda", generator=g) < case["p"]).to(torch.int32)
        ws_bytes = hhs.scan_workspace_size(n)
        st = {"case": case, "flags": flags, "out": torch.zeros_like(flags), "ws_bytes": ws_bytes,
              "ws": torch.zeros(ws_bytes, dtype=torch.uint8, device="cuda")}
        if kind == "compact":
            st["index"] = torch.zeros_like(flags)
            st["count"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        return st
    if kind == "batch":
        sizes = _sizes(case)
        st = _particles(sizes, [seed * 1000 + i for i in range(len(sizes))], hhs.MASS_EQUAL)
        st["batch"] = hhs.Batch(np.concatenate([[0], np.cumsum(sizes)]), eta=case["eta"])
        return {"case": case, **st}
    n = case["n"]
    st = _particles([n], [seed], case["mass"])
    st["ctx"] = hhs.Context(n, 64, case["eta"], case.get("eps", 0.0))
    if kind == "level":
        st["slow"], st["fast"] = hhs.ParticleSystem(n), hhs.ParticleSystem(n)
        st["ts"] = _block(st["system"], "ts", "ts", n)[0]
        rows = st["start"]
        st["pivot"] = _pivot(_timescales(rows[0:3], rows[3:6], st["mass"], case["eta"]))
        st["part"] = torch.zeros(2, dtype=torch.int32, device="cuda")
    return {"case": case, **st}


# The kicks of mixed precision sum FP32 pair terms, so a mixed step's velocities (and
# timesteps) hold FP32 results in FP64 arrays; they are handed on in FP32. Positions, whose
# drifts are FP64, and everything of an FP64 step are handed on as they are.
def _read(case, values):
    return values.to(torch.float32) if case["prec"] == "mixed" else values


# ------------------------------------------------------------------ run
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "scan":
        hhs.scan_exclusive_i32(state["flags"].data_ptr(), state["out"].data_ptr(), case["n"],
                               state["ws"].data_ptr(), state["ws_bytes"])
        return state["out"]
    if kind == "compact":
        hhs.compact_flags_i32(state["flags"].data_ptr(), state["out"].data_ptr(),
                              state["index"].data_ptr(), state["count"].data_ptr(), case["n"],
                              state["ws"].data_ptr(), state["ws_bytes"])
        return [state["out"], state["index"], state["count"]]
    prec = PREC[case["prec"]]
    state["all"].copy_(state["start"])
    if kind == "batch":
        state["batch"].step(state["system"], DT, True, prec)
        return [state["pos"], _read(case, state["vel"])]
    if kind == "hold":
        hhs.hold_step(state["ctx"], state["system"], case["n"], 0.0, DT, True, prec)
        return [state["pos"], _read(case, state["vel"])]
    # one level (src/hold.cuh:100-170): the slow set drifts half a step, the kicks act both
    # ways, the slow set drifts again; the sets are written back to the parent system
    ctx, total, slow, fast = (state[k] for k in ("ctx", "system", "slow", "fast"))
    hhs.timesteps(ctx, total, case["n"], prec)
    hhs.split(ctx, total, slow, fast, state["pivot"], case["n"], state["part"].data_ptr())
    n_slow, n_fast = state["part"].tolist()
    hhs.drift(slow, DT, 0.5, n_slow)
    hhs.kick_slow(slow, DT, 1.0, n_slow, prec)
    hhs.kick_sf(fast, slow, DT, 1.0, n_slow, n_fast, prec)
    hhs.kick_sf(slow, fast, DT, 1.0, n_fast, n_slow, prec)
    hhs.drift(slow, DT, 0.5, n_slow)
    hhs.update_system(total, fast, n_fast)
    hhs.update_system(total, slow, n_slow)
    return [state["pos"], _read(case, state["vel"]), _read(case, state["ts"])]


# ------------------------------------------------------------------ work
PAIR_FLOPS = 20.0  # a pair interaction of a direct sum, the usual count


# Pairs of one HOLD step of a Plummer sphere at dt = 1/64, unordered kick pairs plus unordered
# timestep pairs: counted with the step's own counters at 256 to 65536 particles, they are
# within a tenth of 4.7 n^2 (n / 1024)^0.325 at eta = 0.03, and inverse in eta.
def _hold_pairs(eta, mean_power):
    """mean_power: the mean of n^2.325 over the systems."""
    return 4.7 * (0.03 / eta) * mean_power / 1024.0 ** 0.325


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "scan":
        return {"bytes": 8.0 * n, "flops": 0.0}
    if kind == "compact":
        return {"bytes": 8.0 * n + 4.0 * case["p"] * n, "flops": 0.0}
    if kind == "batch":
        sizes = _sizes(case).astype(np.float64)
        return {"bytes": 13.0 * 8.0 * float(sizes.sum()),
                "flops": PAIR_FLOPS * _hold_pairs(case["eta"], float((sizes ** 2.325).sum()))}
    if kind == "level":
        # n^2 / 2 timestep pairs; kick pairs of two thirds slow, a third fast, unordered
        return {"bytes": 14.0 * 8.0 * n, "flops": PAIR_FLOPS * (0.5 + 4.0 / 9.0) * n * n}
    return {"bytes": 13.0 * 8.0 * n, "flops": PAIR_FLOPS * _hold_pairs(case["eta"], n ** 2.325)}


# ------------------------------------------------------------------ exact
# The same step in plain FP64 tensor operations: the timescales of src/timestep.cuh:27-57, the
# attractive kick, and the recursion of src/hold.cuh:51-181.
def _chunks(p, q):
    """Ranges of p rows whose p x q pairs fit in a few GB of temporaries."""
    step = max(1, (1 << 25) // max(1, q))
    return [(i, min(p, i + step)) for i in range(0, p, step)]


def _timescales(x, v, m, eta):
    """Minimum pair timescale of every particle; x, v: 3 x n."""
    n = x.shape[1]
    out = torch.empty(n, dtype=torch.float64, device=x.device)
    one = torch.ones((), dtype=torch.float64, device=x.device)
    for a, b in _chunks(n, n):
        dr = x[:, a:b, None] - x[:, None, :]
        dv = v[:, a:b, None] - v[:, None, :]
        dr2 = dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2]
        dv2 = dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2]
        rv = (dv[0] * dr[0] + dv[1] * dr[1] + dv[2] * dr[2]) / dr2
        del dr, dv
        r = dr2.sqrt()
        mm = m[a:b, None] + m[None, :]
        free = (eta / 2.0 ** 0.5) * r * (r / mm).sqrt()
        d = 3.0 * free * rv * 0.5
        free = free / (1.0 - 0.5 * torch.where(d < 1.0, d, one))
        fly = eta * r / dv2.sqrt()
        d = fly * rv * (1.0 + mm / (dv2 * r))
        fly = fly / (1.0 - 0.5 * torch.where(d < 1.0, d, one))
        tau = torch.fmin(free, fly)
        tau[torch.arange(b - a, device=x.device), torch.arange(a, b, device=x.device)] = 1e30
        out[a:b] = torch.fmin(tau.amin(1), 1e30 * one)
    return out


def _pull(xi, xj, mj, eps2):
    """Accelerations at xi (3 x p) of masses mj at xj (3 x q)."""
    out = torch.empty_like(xi)
    for a, b in _chunks(xi.shape[1], xj.shape[1]):
        d = xj[:, None, :] - xi[:, a:b, None]
        d2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps2
        w = torch.where(d2 > 0.0, mj / (d2 * d2.sqrt()), torch.zeros_like(d2))
        out[:, a:b] = (d * w).sum(2)
    return out


def _split(ts, dt):
    fast = torch.nonzero(ts <= dt).flatten()
    slow = torch.nonzero(ts > dt).flatten()
    if fast.numel() == 1:  # a lone fast particle joins the slow set
        slow, fast = torch.cat([slow, fast]), fast[:0]
    return slow, fast


def _pivot(ts):
    """The step that makes a third of the particles fast, between two timesteps."""
    order, k = ts.sort().values, len(ts) // 3
    return float(0.5 * (order[k - 1] + order[k]))


def _kick_level(x, v, m, slow, fast, dt, eps2):
    x[:, slow] += v[:, slow] * (0.5 * dt)
    xs, ms = x[:, slow].clone(), m[slow]
    pull = _pull(xs, xs, ms, eps2)
    if fast.numel():
        xf = x[:, fast]
        pull += _pull(xs, xf, m[fast], eps2)
        v[:, fast] += _pull(xf, xs, ms, eps2) * dt
    v[:, slow] += pull * dt
    x[:, slow] += v[:, slow] * (0.5 * dt)


def _hold(x, v, m, ts, index, dt, eta, eps2, calc):
    if calc:
        ts[index] = _timescales(x[:, index], v[:, index], m[index], eta)
    slow, fast = (index[k] for k in _split(ts[index], dt))
    if fast.numel():
        _hold(x, v, m, ts, fast, dt / 2, eta, eps2, False)
    if slow.numel():
        _kick_level(x, v, m, slow, fast, dt, eps2)
    if fast.numel():
        _hold(x, v, m, ts, fast, dt / 2, eta, eps2, True)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("scan", "compact") or (kind == "batch" and case["systems"] > 32) or (
            kind == "hold" and case["n"] > 20000):
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "batch":
        sizes = _sizes(case)
        spheres = [hhs.plummer(int(n), seed * 1000 + i) for i, n in enumerate(sizes)]
    else:
        spheres = [hhs.plummer(case["n"], seed, case["mass"])]
    pos, vel = [], []
    for s in spheres:
        x, v = (torch.tensor(np.stack([s[k] for k in keys]), device=device)
                for keys in (("x", "y", "z"), ("vx", "vy", "vz")))
        m = torch.tensor(s["m"], device=device)
        every = torch.arange(len(s["m"]), device=device)
        if kind == "level":
            ts = _timescales(x, v, m, case["eta"])
            slow, fast = _split(ts, _pivot(ts))
            _kick_level(x, v, m, slow, fast, DT, 0.0)
            return [x, v, ts]
        _hold(x, v, m, torch.zeros_like(m), every, DT, case["eta"], case.get("eps", 0.0) ** 2,
              True)
        pos.append(x)
        vel.append(v)
    return [torch.cat(pos, 1), torch.cat(vel, 1)]
