"""Bulk copies against the ordinary stores of the same launch. The persistent step packs records
with ordinary stores and copies them to shared memory through the asynchronous proxy, in the same
launch; barriers order ordinary accesses only, so a proxy fence has to stand on each side of the
grid barrier between them. Its absence shows as a stale record once in a long while at most, so
the order is read from the source; the GPU cases repeat steps that copy every kind of record."""
import os
import re

import numpy as np
import pytest

from conftest import PKG

FENCE = "fence_proxy_async();"


def _engine():
    src = open(os.path.join(PKG, "csrc", "hhs_engine.cu")).read()
    return re.sub(r"//[^\n]*", "", src)


def _body(src, head):
    start = src.index("{", src.index(head))
    depth = 0
    for k in range(start, len(src)):
        depth += {"{": 1, "}": -1}.get(src[k], 0)
        if depth == 0:
            return src[start:k + 1]
    raise AssertionError(head)


def test_every_thread_fences_before_it_arrives_at_the_grid_barrier():
    src = _engine()
    body = _body(src, "bool grid_barrier(const EParams& E, Smem& sm")
    assert FENCE in body and body.index(FENCE) < body.index("__syncthreads();")
    # except after the timestep and kick phases, which pack no records
    assert src.count("phase_barrier(E, sm, W, false)") == 2


def test_the_issuing_thread_fences_before_its_copies():
    src = _engine()
    helper = _body(src, "void tile_expect(uint64_t* bar, unsigned bytes)")
    assert helper.index(FENCE) < helper.index("mbar_arrive_expect_tx(")
    # copies are announced by that helper and by nothing else, right before they are issued
    assert src.count("mbar_arrive_expect_tx(") == 1
    copies = [m.start() for m in re.finditer(r"\bbulk_load\(", src)]
    assert len(copies) >= 3
    for c in copies:
        before = src[:c]
        assert "tile_expect(" in before[before.rindex("__device__"):] or \
            "tile_expect(" in before[before.rindex("auto stage = [&]() {"):]


# mixed: kick records and full timestep records (4099), filter records too (17001); FP64: filter
# records only
@pytest.mark.gpu
@pytest.mark.parametrize("n,prec,passes", [(4099, 1, 40), (17001, 1, 20), (4099, 0, 20)])
def test_repeated_steps_have_the_same_bits(cuda, hhs, n, prec, passes):
    s = hhs.plummer(n, 3, 1)
    d = hhs.ParticleSystem(n)
    ctx = hhs.Context(n, 64, 0.02)
    first = None
    for _ in range(passes):
        d.upload(s)
        hhs.hold_step(ctx, d, n, 0.0, 1.0 / 64, True, prec)
        ctx.check()
        out = d.download()
        first = first or out
        for k in ("x", "y", "z", "vx", "vy", "vz", "ts"):
            assert np.array_equal(out[k], first[k]), k
