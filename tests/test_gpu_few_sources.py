"""Kicks of many sinks by few sources, where a thread takes a sink: around the rule's line and
against the time per source that it is meant to keep."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _systems(hhs, n_sink, n_src):
    def cut(n, seed):
        s = hhs.plummer(max(2, n), seed)
        return {k: np.ascontiguousarray(v[:n]) for k, v in s.items()}

    sink, src = cut(n_sink, 5), cut(n_src, 6)
    for k in ("x", "y", "z"):  # a coincident pair contributes nothing
        sink[k][-1] = src[k][0]
    a, b = hhs.ParticleSystem(n_sink), hhs.ParticleSystem(n_src)
    a.upload(sink)
    b.upload(src)
    return sink, src, a, b


SHAPES = [(4096, 1), (4097, 33), (4096, 64), (10000, 95), (32768, 1), (32769, 129), (32768, 400),
          (32768, 700), (100000, 20)]


@pytest.mark.parametrize("n_sink,n_src", SHAPES)
def test_fp64_equals_oracle(cuda, hhs, oracle, n_sink, n_src):
    sink, src, a, b = _systems(hhs, n_sink, n_src)
    hhs.kick_sf(b, a, 0.01, 1.0, n_sink, n_src, hhs.PREC_FP64)
    got = a.download()
    oracle.kick(sink, src, 0.01)
    for k in ("vx", "vy", "vz"):
        assert np.array_equal(got[k], sink[k]), k


@pytest.mark.parametrize("n_sink,n_src", SHAPES)
def test_mixed_within_the_bound_of_its_terms(cuda, hhs, oracle, n_sink, n_src):
    sink, src, a, b = _systems(hhs, n_sink, n_src)
    hhs.kick_sf(b, a, 1.0, 1.0, n_sink, n_src, hhs.PREC_MIXED)
    got = a.download()
    dv = np.stack([got[k] - sink[k] for k in ("vx", "vy", "vz")])
    # the sum of the pair terms' magnitudes, times the bound of a mixed pair term
    r2 = sum((src[k][None, :] - sink[k][:, None]) ** 2 for k in ("x", "y", "z"))
    mag = np.where(r2 > 0, src["m"][None, :] / np.where(r2 > 0, r2, 1.0), 0.0).sum(1)
    acc = oracle.kick(sink, src, 1.0)
    assert np.all(np.abs(dv - acc) <= 5e-7 * mag + 1e-15)


@pytest.mark.parametrize("prec", [0, 1])
def test_time_of_few_sources(cuda, hhs, prec):
    """100000 sinks and 10 sources: with a CTA for 8 or 32 sinks 123 us in FP64, 18 mixed."""
    _, _, a, b = _systems(hhs, 100000, 10)
    best = 1e30
    for _ in range(10):
        e0, e1 = (cuda.cuda.Event(enable_timing=True) for _ in range(2))
        cuda.cuda.synchronize()
        e0.record()
        for _ in range(20):
            hhs.kick_sf(b, a, 1e-9, 1.0, 100000, 10, prec)
        e1.record()
        cuda.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1) / 20)
    assert best < (0.04 if prec == 0 else 0.014)
