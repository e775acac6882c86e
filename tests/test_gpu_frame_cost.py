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
