"""The filters of the timesteps take the same time in any frame: their tests use squares of
positions and velocities, whose rounding would let pairs pass when the whole system is displaced
or moves. Times of one process on one device, least of several; the bounds are far above the
spread of such times and far below what a filter that passes every pair takes (6 to 30 times)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(hhs, n, shift, velocity):
    s = hhs.plummer(n, 5)
    s["x"] += shift
    s["vy"] += velocity
    return s


def _least_ms(torch, call, reset, repeats=5):
    best = 1e30
    for _ in range(repeats + 1):
        reset()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        call()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [2051, 16384])
def test_timesteps_call(cuda, hhs, n, prec):
    def ms(shift, velocity):
        d = hhs.ParticleSystem(n)
        d.upload(_system(hhs, n, shift, velocity))
        ctx = hhs.Context(n, 8, 0.03)
        return _least_ms(cuda, lambda: hhs.timesteps(ctx, d, n, prec), lambda: None)

    plain = ms(0.0, 0.0)
    assert ms(1000.0, 0.0) < 1.5 * plain + 0.01
    assert ms(0.0, 200.0) < 1.5 * plain + 0.01


def _pair_of_clusters(hhs, n, distance):
    s = hhs.plummer(n, 5)
    s["x"][n // 2:] += distance
    return s


@pytest.mark.parametrize("kind,n", [("eta", 16384), ("clusters", 16384), ("eta", 4097)])
def test_timesteps_call_that_the_filter_does_not_help(cuda, hhs, kind, n):
    """Every pair passes (the test's range ends at eta = 1), or half of them do (two clusters far
    apart): the evaluation of every pair without a test takes 3 times the filtered call's."""
    def ms(s, eta):
        d = hhs.ParticleSystem(n)
        d.upload(s)
        ctx = hhs.Context(n, 8, eta)
        return _least_ms(cuda, lambda: hhs.timesteps(ctx, d, n, hhs.PREC_MIXED), lambda: None)

    plain = ms(hhs.plummer(n, 5), 0.03)
    other = ms(hhs.plummer(n, 5), 1.5) if kind == "eta" else ms(_pair_of_clusters(hhs, n, 1e3), 0.03)
    assert other < 4.5 * plain


@pytest.mark.parametrize("n", [3, 511, 513, 4097, 9999])
def test_dense_tiles(cuda, hhs, oracle, n):
    """Two clusters far apart, member by member: tiles of which half the pairs pass. Positions on a
    grid of 2^-20 lengths are exact in double-single form at a distance of 2^12, so the bound of
    the mixed timesteps holds; eta beyond the test's range passes all."""
    s = hhs.plummer(n, 7)
    for k in ("x", "y", "z"):
        s[k] = np.round(s[k] * 2.0 ** 20) / 2.0 ** 20
    s["x"][1::2] += 4096.0
    for eta in (0.03, 1.5):
        d = hhs.ParticleSystem(n)
        d.upload(s)
        hhs.timesteps(hhs.Context(n, 8, eta), d, n, hhs.PREC_MIXED)
        ref = oracle.timesteps(s, eta)
        assert np.all(np.abs(d.download()["ts"] - ref) <= 2e-6 * ref)


@pytest.mark.parametrize("prec", [0, 1])
def test_step(cuda, hhs, prec):
    """The phase that computes timesteps in a step, whose pairs the same filter tests. (A shift by
    a power of two and a rounded start keep the displaced system the same system.)"""
    n = 9001

    def ms(shift, velocity):
        s = hhs.plummer(n, 5)
        for k in ("x", "y", "z", "vx", "vy", "vz"):
            s[k] = np.round(s[k] * 2.0 ** 32) / 2.0 ** 32
        s["x"] += shift
        s["vy"] += velocity
        d = hhs.ParticleSystem(n)
        ctx = hhs.Context(n, 64, 0.03)
        ctx.set_profiling(True)
        best, before = 1e30, 0.0
        for _ in range(4):
            d.upload(s)
            hhs.hold_step(ctx, d, n, 0.0, 1.0 / 64, True, prec)
            ctx.check()
            total = ctx.profile()["timesteps"]["ms"]
            best, before = min(best, total - before), total
        return best

    plain = ms(0.0, 0.0)
    assert ms(1024.0, 0.0) < 1.5 * plain
    assert ms(0.0, 256.0) < 1.5 * plain


def _units(hhs, n):
    """A cluster in units of 1e-7 of its size and 1e14 of its time."""
    s = hhs.plummer(n, 5)
    for k in ("x", "y", "z"):
        s[k] *= 1e7
    for k in ("vx", "vy", "vz"):
        s[k] *= 1e-7
    s["m"] *= 1e-7
    return s, 1e14 / 64


def _disk(hhs, n):
    """Light members on nearly circular orbits about one mass."""
    s = hhs.plummer(n, 5)
    r = np.random.default_rng(5)
    a, ph, dv = r.uniform(1, 2, n), r.uniform(0, 2 * np.pi, n), r.normal(size=(3, n)) * 1e-2
    s["x"][:], s["y"][:], s["z"][:] = a * np.cos(ph), a * np.sin(ph), r.normal(size=n) * 1e-2
    s["vx"][:] = dv[0] - np.sin(ph) / np.sqrt(a)
    s["vy"][:] = dv[1] + np.cos(ph) / np.sqrt(a)
    s["vz"][:] = dv[2]
    s["m"][:] = 1e-9
    s["m"][0] = 1.0
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        s[k][0] = 0.0
    return s, 1.0 / 64


def _phases(hhs, s, dt, eta, prec):
    n = len(s["x"])
    d = hhs.ParticleSystem(n)
    ctx = hhs.Context(n, 64, eta)
    ctx.set_profiling(True)
    best, before = None, None
    for _ in range(4):
        d.upload(s)
        hhs.hold_step(ctx, d, n, 0.0, dt, True, prec)
        ctx.check()
        p = {k: v["ms"] for k, v in ctx.profile().items() if isinstance(v, dict) and "ms" in v}
        now = p if before is None else {k: p[k] - before[k] for k in p}
        best = now if best is None else {k: min(best[k], now[k]) for k in p}
        before = p
    return best


def test_step_in_other_units(cuda, hhs):
    """No pair can be left out where the test's numbers leave their range: the timestep phase then
    takes the evaluation of every pair, twice the filtered one's time (30 times through lists)."""
    n = 16384
    plain = _phases(hhs, hhs.plummer(n, 5), 1.0 / 64, 0.03, hhs.PREC_MIXED)["timesteps"]
    s, dt = _units(hhs, n)
    assert _phases(hhs, s, dt, 0.03, hhs.PREC_MIXED)["timesteps"] < 3.0 * plain


@pytest.mark.parametrize("n", [6001, 9001, 16384])
@pytest.mark.parametrize("kind", ["units", "disk"])
def test_step_without_the_filter_where_it_does_not_help(cuda, hhs, kind, n):
    """The same bits as the step from equal timesteps, which is never filtered."""
    s, dt = _units(hhs, n) if kind == "units" else _disk(hhs, n)
    a, b = hhs.ParticleSystem(n), hhs.ParticleSystem(n)
    ctx = hhs.Context(n, 64, 0.03)
    a.upload(s)
    b.upload(s)
    hhs.hold_step(ctx, a, n, 0.0, dt, True, hhs.PREC_MIXED)
    ctx.check()
    hhs.timesteps(ctx, b, n, hhs.PREC_MIXED)
    hhs.hold_step(ctx, b, n, 0.0, dt, False, hhs.PREC_MIXED)
    ctx.check()
    x, y = a.download(), b.download()
    for k in ("x", "y", "z", "vx", "vy", "vz", "ts"):
        assert np.array_equal(x[k], y[k]), k


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("eta", [0.25, 0.5, 1.0])
def test_step_with_large_timesteps(cuda, hhs, eta, prec):
    """Rates change with eta from one calculation to the next; a row whose bound was too high is
    scanned whole in the split phase, which then took 30 to 80% of the step (it takes 4 to 6%)."""
    p = _phases(hhs, hhs.plummer(9001, 5), 0.125 if eta < 1.0 else 0.25, eta, prec)
    assert p["split"] < 0.15 * sum(p.values())


@pytest.mark.parametrize("n", [1001, 2500])
def test_rows_whose_bound_was_too_high_fp64(cuda, hhs, oracle, n):
    """A common velocity of 2^20 leaves FP32 relative velocities of 2^-4: the bounds of the top
    node, from FP32 rates, exceed many FP64 rates, and the rows are scanned whole."""
    s = hhs.plummer(n, 5)
    s["vy"] += 2.0 ** 20
    ts = oracle.timesteps(s, 0.03)
    d = hhs.ParticleSystem(n)
    d.upload(s)
    ctx = hhs.Context(n, 64, 0.03)
    hhs.timesteps(ctx, d, n, hhs.PREC_MIXED)  # the same FP32 rates
    assert np.count_nonzero(0.999 / d.download()["ts"] * ts > 1.0) > n // 20
    d.upload(s)
    hhs.hold_step(ctx, d, n, 0.0, 1.0 / 64, True, hhs.PREC_FP64)
    ctx.check()
    oracle.hold_step(s, 1.0 / 64, True, 0.03)
    out = d.download()
    for k in ("x", "y", "z", "vx", "vy", "vz", "ts"):
        assert np.array_equal(out[k], s[k]), k


def test_step_in_other_units_small_nodes(cuda, hhs):
    """A step whose nodes are mostly below 1024 members: 1.5 times the filtered phase (3.3 times when
    those went through lists)."""
    n = 12000
    plain = _phases(hhs, hhs.plummer(n, 5), 1.0 / 64, 0.03, hhs.PREC_MIXED)["timesteps"]
    s, dt = _units(hhs, n)
    assert _phases(hhs, s, dt, 0.03, hhs.PREC_MIXED)["timesteps"] < 2.4 * plain
