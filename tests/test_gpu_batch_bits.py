"""A mixed system's bits in a batch follow from the system, not from the others of the batch (whose
sizes decide how many CTAs work on it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "vx", "vy", "vz", "ts")


def _step(hhs, sizes, tuning=None):
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    parts = [hhs.plummer(n, n) for n in sizes]
    d = hhs.ParticleSystem(int(off[-1]))
    d.upload({k: np.concatenate([p[k] for p in parts]) for k in parts[0]})
    b = hhs.Batch(off, 64, 0.03)
    if tuning:
        b.set_tuning(**tuning)
    for _ in range(2):
        b.step(d, 1.0 / 64, True, hhs.PREC_MIXED)
    b.check()
    out = d.download()
    return {k: out[k][:sizes[0]].copy() for k in KEYS}


@pytest.mark.parametrize("n", [641, 800, 1024, 1025, 2049, 3001])
def test_bits_do_not_depend_on_the_other_systems(cuda, hhs, n):
    # alone: clusters of 16; 12 more of its size: of 8; 48 more: of 4 (a CTA each for those of at
    # most 1024 beside a larger one)
    alone = _step(hhs, [n])
    for others in ([n] * 12, [n] * 48, [3001], [4001, 100]):
        other = _step(hhs, [n] + others)
        for k in KEYS:
            assert np.array_equal(alone[k], other[k]), (k, len(others))


def test_many_small_systems_take_no_longer_than_a_cta_each(cuda, hhs):
    """Default tuning against every system on a CTA of its own, where more systems exceed 640
    particles than there are clusters and many smaller ones wait behind them."""
    r = np.random.default_rng(3)
    sizes = np.exp(r.uniform(np.log(64), np.log(1024), 500)).astype(int)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    parts = [hhs.plummer(int(n), int(n)) for n in sizes]
    s = {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}
    d = hhs.ParticleSystem(int(off[-1]))
    default, each = hhs.Batch(off, 64, 0.03), hhs.Batch(off, 64, 0.03)
    each.set_tuning(big_n=1024)
    best = {default: 1e30, each: 1e30}
    for b in [default, each] * 12:
        d.upload(s)
        e0, e1 = (cuda.cuda.Event(enable_timing=True) for _ in range(2))
        cuda.cuda.synchronize()
        e0.record()
        b.step(d, 1.0 / 64, True, hhs.PREC_MIXED)
        e1.record()
        cuda.cuda.synchronize()
        b.check()
        best[b] = min(best[b], e0.elapsed_time(e1))
    assert best[default] < 1.15 * best[each]


def test_scratch_of_a_batch(cuda, hhs):
    """A slot holds the kick's partial sums (32 chunks of three components) and the level lists, and
    every CTA and cluster of the launch has one: no partial timesteps (a quarter more)."""
    n, slots = 4096, 148 * 2 + 148 * 2 // 4
    b = hhs.Batch(np.array([0, 64], dtype=np.int32), 1, 0.03)  # loads the kernel
    cuda.cuda.synchronize()
    free = cuda.cuda.mem_get_info()[0]
    c = hhs.Batch(np.array([0, n], dtype=np.int32), 1, 0.03)
    used = free - cuda.cuda.mem_get_info()[0]
    per_slot = n * (32 * 3 * 8 + 2 * 4 + 4) + 4096
    assert used <= slots * per_slot + (4 << 20)
    c.destroy()
    b.destroy()


def test_autotune_keeps_to_its_precision(cuda, hhs):
    """The tuner times the batch's own big_n among its candidates, the default too, and sets that of
    the precision it times only."""
    sizes = [700, 900, 64, 300]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    parts = [hhs.plummer(n, n) for n in sizes]
    d = hhs.ParticleSystem(int(off[-1]))
    d.upload({k: np.concatenate([p[k] for p in parts]) for k in parts[0]})
    b = hhs.Batch(off, 64, 0.03)
    for prec in (hhs.PREC_FP64, hhs.PREC_MIXED):
        assert 640 in {t["big_n"] for t in b.autotune(d, 1.0 / 64, prec)[1]}
    b.set_tuning(big_n=800)
    b.autotune(d, 1.0 / 64, hhs.PREC_MIXED)
    assert 800 in {t["big_n"] for t in b.autotune(d, 1.0 / 64, hhs.PREC_FP64)[1]}
