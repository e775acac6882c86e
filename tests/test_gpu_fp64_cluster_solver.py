"""FP64 subtrees of 97 to 640 members on clusters: the device step runs them on the whole grid, the
batched step on its clusters of 4, 8 or 16 CTAs, with the nodes above mid_dist_n divided over them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [0, 12, 48], ids=["clusters of 16", "of 8", "of 4"])
@pytest.mark.parametrize("n,mid_n,dist_n,spectrum", [(700, 640, 96, 0), (700, 640, 0, 1),
                                                     (1500, 640, 16, 0), (1300, 256, 32, 2)])
def test_batched_clusters_equal_oracle(cuda, hhs, oracle, n, mid_n, dist_n, spectrum, copies):
    parts = [hhs.plummer(n, 11, spectrum), hhs.plummer(641, 12, spectrum)]
    parts += [hhs.plummer(n, 13, spectrum)] * copies
    off = np.concatenate([[0], np.cumsum([len(p["x"]) for p in parts])]).astype(np.int32)
    d = hhs.ParticleSystem(int(off[-1]))
    d.upload({k: np.concatenate([p[k] for p in parts]) for k in parts[0]})
    b = hhs.Batch(off, 64, 0.03)
    b.set_mid(mid_n, dist_n)
    b.step(d, 1.0 / 64, True, hhs.PREC_FP64)
    b.check()
    out = d.download()
    for i, p in enumerate(parts[:3]):
        ref = {k: v.copy() for k, v in p.items()}
        oracle.hold_step(ref, 1.0 / 64, True, 0.03)
        for k in ("x", "y", "z", "vx", "vy", "vz", "ts"):
            assert np.array_equal(out[k][off[i]:off[i + 1]], ref[k]), (i, k)
