"""The filtered timesteps of the device step: nodes below the top one pass over their pairs with a
test and evaluate only those that pass, so the step has to equal one that evaluates every pair.
FP64: the oracle, bit for bit. Mixed: the step from equal timesteps without the filter
(calc_timestep = False keeps it off; the timesteps are then computed by the standalone call)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cluster(hhs, n, seed, mass, kind):
    s = hhs.plummer(n, seed, mass)
    rng = np.random.default_rng(seed)
    if kind == "binaries":  # close pairs: rates far above the others' (and bounds that fail)
        k = 12
        for c in ("x", "y", "z"):
            s[c][:k] = s[c][k:2 * k] + rng.normal(size=k) * 1.5e-3
        for c in ("vx", "vy", "vz"):
            s[c][:k] = s[c][k:2 * k] + rng.normal(size=k) * 0.3
    elif kind == "streams":  # groups with nearly equal velocities: the |dv| test
        for c in ("vx", "vy", "vz"):
            s[c][:] = np.round(s[c], 1) + rng.normal(size=n) * 1e-6
    elif kind == "offset":  # far from the origin: rounding of the dot products
        s["x"] += 300.0
        s["vy"] += 40.0
    return s


@pytest.mark.parametrize("n,mass,eta,kind", [
    (1001, 0, 0.03, "plain"), (2047, 1, 0.02, "plain"), (2049, 2, 0.03, "binaries"),
    (3001, 0, 0.03, "streams"), (2500, 1, 0.9, "plain"), (2500, 0, 1.5, "plain"),
    (4097, 0, 0.03, "offset"), (5000, 1, 0.02, "binaries")])
def test_filtered_step_fp64_equals_oracle(cuda, hhs, oracle, n, mass, eta, kind):
    s = _cluster(hhs, n, 11, mass, kind)
    d = hhs.ParticleSystem(n)
    ctx = hhs.Context(n, 64, eta)
    ctx.set_tuning(mid_n=0 if n < 1500 else 64, small_n=0, warp_n=0 if n < 1500 else 32)
    d.upload(s)
    dt = 1.0 / 64 if eta < 0.5 else 0.25
    for _ in range(2):
        hhs.hold_step(ctx, d, n, 0.0, dt, True, hhs.PREC_FP64)
        ctx.check()
        oracle.hold_step(s, dt, True, eta)
    out = d.download()
    for k in ("x", "y", "z", "vx", "vy", "vz", "ts"):
        assert np.array_equal(out[k], s[k]), k


@pytest.mark.parametrize("n,mass,kind", [(5999, 0, "plain"), (6001, 1, "binaries"),
                                         (16384, 0, "plain"), (17001, 2, "streams"),
                                         (9000, 0, "offset")])
def test_filtered_step_mixed_equals_the_unfiltered_one(cuda, hhs, n, mass, kind):
    s = _cluster(hhs, n, 5, mass, kind)
    a, b = hhs.ParticleSystem(n), hhs.ParticleSystem(n)
    ctx = hhs.Context(n, 64, 0.03)
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
