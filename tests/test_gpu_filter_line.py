"""Where mixed steps begin to filter their timesteps (10000 particles): the same bits as steps without
the filter on both sides, and a kernel without it below, whose other phases are faster."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(hhs, n, kind):
    s = hhs.plummer(n, 5, 1 if kind == "binaries" else 0)
    r = np.random.default_rng(n)
    if kind == "binaries":
        k = 12
        for c in ("x", "y", "z"):
            s[c][:k] = s[c][k:2 * k] + r.normal(size=k) * 1.5e-3
        for c in ("vx", "vy", "vz"):
            s[c][:k] = s[c][k:2 * k] + r.normal(size=k) * 0.3
    elif kind == "moving":
        s["x"] += 300.0
        s["vy"] += 40.0
    elif kind == "heavy":
        s["m"][7] = 1.0
    elif kind == "units":
        for c in ("x", "y", "z"):
            s[c] *= 1e7
        for c in ("vx", "vy", "vz"):
            s[c] *= 1e-7
        s["m"] *= 1e-7
    return s, (1e14 if kind == "units" else 1.0) / 64


@pytest.mark.parametrize("n", [9999, 10000, 10001, 12289])
@pytest.mark.parametrize("kind", ["plain", "binaries", "moving", "heavy", "units"])
def test_step_equals_the_unfiltered_one(cuda, hhs, kind, n):
    s, dt = _system(hhs, n, kind)
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


def test_collapse_below_the_line(cuda, hhs):
    """No velocities: deep subtrees, hardly any grid timesteps. Their time with and without the
    timesteps' computation at the top (which the filter's kernel needs, and whose solver took 8%
    longer) differs by that alone."""
    n = 9000
    s = hhs.plummer(n, 5)
    for k in ("vx", "vy", "vz"):
        s[k][:] = 0.0
    d = hhs.ParticleSystem(n)
    ctx = hhs.Context(n, 64, 0.03)
    ctx.set_profiling(True)
    best, before = [1e30, 1e30], ctx.profile().get("cluster_node", {"ms": 0.0})["ms"]
    for _ in range(6):
        for calc in (0, 1):
            d.upload(s)
            if not calc:
                hhs.timesteps(ctx, d, n, hhs.PREC_MIXED)
            hhs.hold_step(ctx, d, n, 0.0, 1.0 / 64, bool(calc), hhs.PREC_MIXED)
            ctx.check()
            now = ctx.profile()["cluster_node"]["ms"]
            best[calc], before = min(best[calc], now - before), now
    assert best[1] < 1.04 * best[0]


@pytest.mark.parametrize("small_n,mid_n", [(64, 0), (700, 640), (128, 100), (640, 640)])
def test_tunings_with_single_cta_nodes(cuda, hhs, small_n, mid_n):
    """Nodes that the tuning gives to one CTA, above the subtree solver's size: steps without the
    filter, which has no code for them. The same bits as from equal timesteps."""
    n = 10007
    s = hhs.plummer(n, 5)
    a, b = hhs.ParticleSystem(n), hhs.ParticleSystem(n)
    ctx = hhs.Context(n, 64, 0.03)
    ctx.set_tuning(small_n=small_n, mid_n=mid_n)
    a.upload(s)
    b.upload(s)
    hhs.hold_step(ctx, a, n, 0.0, 1.0 / 64, True, hhs.PREC_MIXED)
    ctx.check()
    hhs.timesteps(ctx, b, n, hhs.PREC_MIXED)
    hhs.hold_step(ctx, b, n, 0.0, 1.0 / 64, False, hhs.PREC_MIXED)
    ctx.check()
    x, y = a.download(), b.download()
    for k in ("x", "y", "z", "vx", "vy", "vz", "ts"):
        assert np.array_equal(x[k], y[k]), k
