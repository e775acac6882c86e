"""The reference-shaped timesteps and mixed kicks at the edges of their tiles: timesteps of 8, 16 and
32 rows a CTA against tiles of 512 columns, kicks of 32 sinks against 8 x 32 sources."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _upload(hhs, s):
    d = hhs.ParticleSystem(len(s["x"]))
    d.upload(s)
    return d


@pytest.mark.parametrize("n,kind,eta", [
    (1, "plain", 0.03), (3, "plain", 0.03), (33, "coincident", 0.03), (511, "plain", 0.02),
    (513, "cold", 0.03), (4736, "plain", 0.03), (4737, "heavy", 0.02), (9473, "plain", 0.03),
    (2000, "offset", 0.03), (1500, "plain", 1.5)])
def test_timesteps_tile_edges(cuda, hhs, oracle, n, kind, eta):
    s = hhs.plummer(max(2, n), 3, 1 if kind == "heavy" else 0)
    s = {k: np.ascontiguousarray(v[:n]) for k, v in s.items()}
    if kind == "coincident":  # timestep 0, and every pair of those two rows passes the test
        for k in ("x", "y", "z"):
            s[k][5] = s[k][20]
    elif kind == "cold":      # no relative velocity: free-fall times only
        for k in ("vx", "vy", "vz"):
            s[k][:] = 0.0
    elif kind == "offset":
        s["x"] += 1000.0
    ctx = hhs.Context(n, 8, eta)
    d = _upload(hhs, s)
    hhs.timesteps(ctx, d, n, hhs.PREC_FP64)
    ref = oracle.timesteps(s, eta)
    assert np.array_equal(d.download()["ts"], ref)
    hhs.timesteps(ctx, d, n, hhs.PREC_MIXED)
    out = d.download()["ts"]
    ok = ref > 0
    # the bound of the mixed timesteps; far from the origin the double-single positions carry
    # 2^-48 of 1000, against pair distances of 1e-2
    tol = 2e-6 if kind != "offset" else 2e-5
    assert np.all(np.abs(out[ok] - ref[ok]) <= tol * ref[ok]) and np.all(out[~ok] == 0.0)


@pytest.mark.parametrize("n_sink,n_src", [(1, 1), (31, 255), (32, 256), (33, 257), (65, 3),
                                          (500, 1000)])
def test_kick_sf_mixed_tile_edges(cuda, hhs, oracle, n_sink, n_src):
    sink, src = hhs.plummer(max(2, n_sink), 5), hhs.plummer(max(2, n_src), 6)
    sink = {k: np.ascontiguousarray(v[:n_sink]) for k, v in sink.items()}
    src = {k: np.ascontiguousarray(v[:n_src]) for k, v in src.items()}
    for k in ("x", "y", "z"):  # coincident pairs contribute nothing
        sink[k][-1] = src[k][0]
    a, b = _upload(hhs, sink), _upload(hhs, src)
    hhs.kick_sf(b, a, 1.0, 1.0, n_sink, n_src, hhs.PREC_MIXED)
    got = a.download()
    dv = np.stack([got[k] - sink[k] for k in ("vx", "vy", "vz")])
    # the sum of the pair terms' magnitudes, times the bound of a mixed pair term
    d = [src[k][None, :] - sink[k][:, None] for k in ("x", "y", "z")]
    r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
    mag = np.where(r2 > 0, src["m"][None, :] / np.where(r2 > 0, r2, 1.0), 0.0).sum(1)
    acc = oracle.kick(sink, src, 1.0)
    assert np.all(np.abs(dv - acc) <= 5e-7 * mag + 1e-15)


@pytest.mark.parametrize("n", [2, 7, 8, 31, 32, 63, 64, 65])
@pytest.mark.parametrize("eta", [0.03, 1.5])
def test_timesteps_of_few_particles(cuda, hhs, oracle, n, eta):
    """Up to 64 particles every pair is evaluated without a test."""
    s = hhs.plummer(n, 3)
    ctx = hhs.Context(n, 8, eta)
    d = _upload(hhs, s)
    ref = oracle.timesteps(s, eta)
    hhs.timesteps(ctx, d, n, hhs.PREC_FP64)
    assert np.array_equal(d.download()["ts"], ref)
    hhs.timesteps(ctx, d, n, hhs.PREC_MIXED)
    assert np.all(np.abs(d.download()["ts"] - ref) <= 2e-6 * ref)


def test_timesteps_of_few_particles_take_less_than_of_many(cuda, hhs):
    """Mixed: 16 particles against 256, whose rows go through the test's phases (as those of 16 did)."""
    def us(n):
        d = _upload(hhs, hhs.plummer(n, 3))
        ctx = hhs.Context(n, 8, 0.03)
        best = 1e30
        for _ in range(10):
            e0, e1 = (cuda.cuda.Event(enable_timing=True) for _ in range(2))
            cuda.cuda.synchronize()
            cuda.cuda._sleep(400000)
            e0.record()
            for _ in range(50):
                hhs.timesteps(ctx, d, n, hhs.PREC_MIXED)
            e1.record()
            cuda.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1) * 20.0)
        return best

    assert us(16) < 0.75 * us(256)
