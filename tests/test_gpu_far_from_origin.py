"""Systems far from the origin of their coordinates (a galactocentric position in metres, say):
padding that stands at the origin must not reach a result, since a pair with it overflows FP32
where no pair of the system does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FAR, LENGTH, MASS = 2.5e20, 1e14, 1e30  # offset, size and total mass
# a coordinate in double-single form keeps 48 bits: 2^-49 of it is lost at most, by either particle
# of a pair, in three coordinates
LOST = 2.0 * 3.0 ** 0.5 * 2.0 ** -49 * FAR


def _far(hhs, n, seed):
    s = hhs.plummer(max(2, n), seed)
    s = {k: np.ascontiguousarray(v[:n]) for k, v in s.items()}
    for k in ("x", "y", "z"):
        s[k] *= LENGTH
    s["x"] += FAR
    s["m"][:] = MASS / n
    return s


def _pair_sums(sink, src):
    """Per sink: the sums of the pair terms' magnitudes m / r^2 and of their slopes 2 m / r^3."""
    d = [src[k][None, :] - sink[k][:, None] for k in ("x", "y", "z")]
    r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
    r2 = np.where(r2 > 0, r2, np.inf)
    return (src["m"] / r2).sum(1), (2.0 * src["m"] / r2 ** 1.5).sum(1)


@pytest.mark.parametrize("n_sink,n_src", [(1, 1), (33, 9), (40, 255), (65, 257), (100, 1001)])
def test_kick_sf_mixed_odd_slices(cuda, hhs, oracle, n_sink, n_src):
    sink, src = _far(hhs, n_sink, 5), _far(hhs, n_src, 6)
    a, b = hhs.ParticleSystem(n_sink), hhs.ParticleSystem(n_src)
    a.upload(sink)
    b.upload(src)
    hhs.kick_sf(b, a, 1.0, 1.0, n_sink, n_src, hhs.PREC_MIXED)
    got = a.download()
    dv = np.stack([got[k] - sink[k] for k in ("vx", "vy", "vz")])
    mag, slope = _pair_sums(sink, src)
    acc = oracle.kick(sink, src, 1.0)
    # the bound of a mixed pair term, and what the positions lose
    assert np.all(np.abs(dv - acc) <= 5e-7 * mag + LOST * slope)


@pytest.mark.parametrize("n", [20, 100, 2500])
def test_fp64_timestep_of_a_coincident_pair_of_negative_mass(cuda, hhs, oracle, n):
    """Its timescale is -0, below every other, and every calculation of the pair gives it."""
    s = hhs.plummer(n, 5)
    for k in ("x", "y", "z"):
        s[k][3] = s[k][n - 2]
    s["m"][3] = -2.0 * s["m"][n - 2]
    ref = oracle.timesteps(s, 0.03)
    assert ref[3] == 0.0 and ref[n - 2] == 0.0
    d = hhs.ParticleSystem(n)
    d.upload(s)
    hhs.timesteps(hhs.Context(n, 8, 0.03), d, n, hhs.PREC_FP64)
    got = d.download()["ts"]
    assert got[3] == 0.0 and got[n - 2] == 0.0
    assert np.array_equal(got, ref)
