"""FP64 kick of a block of sinks (hhs_kick64.cuh) at the edges of its tiles: the pair terms are
evaluated by a whole CTA and added in source order, so every sum equals the oracle's bit for
bit (blocks of 8 sinks x stages of 224 sources)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sink,n_src", [(1, 1), (7, 223), (8, 224), (9, 225), (8, 449),
                                          (33, 1000), (16384, 17), (16385, 63), (16417, 129)])
def test_kick_sf_fp64_tile_edges_bit_exact(cuda, hhs, oracle, n_sink, n_src):
    sink, src = hhs.plummer(max(2, n_sink), 5), hhs.plummer(max(2, n_src), 6)
    sink = {k: np.ascontiguousarray(v[:n_sink]) for k, v in sink.items()}
    src = {k: np.ascontiguousarray(v[:n_src]) for k, v in src.items()}
    # coincident pairs contribute nothing
    for k in ("x", "y", "z"):
        sink[k][-1] = src[k][0]
        sink[k][0] = src[k][-1]
    a, b = hhs.ParticleSystem(n_sink), hhs.ParticleSystem(n_src)
    a.upload(sink)
    b.upload(src)
    hhs.kick_sf(b, a, 0.01, 1.0, n_sink, n_src, hhs.PREC_FP64)
    got = a.download()
    oracle.kick(sink, src, 0.01)
    for k in ("vx", "vy", "vz"):
        assert np.array_equal(got[k], sink[k]), k
