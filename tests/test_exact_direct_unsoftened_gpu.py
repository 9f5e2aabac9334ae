"""The exact direct sum without softening and with masses or positions out of
the branch-free weight's range: bit-identical at the edges of the block
layouts, and in the time of one form of the weight, not of both."""
import time

import numpy as np
import pytest

import oracle
import physgpu.ics as ics
from physgpu import DIRECT, F64_EXACT, make_params

pytestmark = pytest.mark.gpu


def bodies(kind, n):
    pos, vel, m = ics.plummer(n, seed=n)
    eps = 0.0
    if kind == "close":  # a separation below the range, in one chunk
        pos[n - 2], pos[n - 1] = [1e-35, 0.0, -1e-36], [-2e-35, 1e-35, 0.0]
    elif kind == "small":  # every separation below it
        pos *= 1e-40
        m *= 1e-60
    elif kind == "masses":
        m *= 1e-100
        eps = 0.01
    elif kind == "one":
        m[n // 2] = 1e90
        pos[n // 3] *= 1e33
        eps = 0.01
    return pos, vel, m, eps


@pytest.mark.parametrize("kind", ["plain", "close", "small", "masses", "one"])
@pytest.mark.parametrize("n", [3, 33, 129, 1185, 2367, 2368, 2369, 2401])
def test_bits(ctx, kind, n):
    pos, vel, m, eps = bodies(kind, n)
    p = make_params(1.0, eps, method=DIRECT, precision=F64_EXACT)
    ctx.upload(pos, vel, m)
    assert np.array_equal(ctx.gravity_forces(p), oracle.direct_forces(pos, m, 1.0, eps))


@pytest.mark.parametrize("n", [40, 2368, 2369])
def test_ticks(ctx, n):
    pos, vel, m, _ = bodies("plain", n)
    ctx.upload(pos, vel, m)
    ctx.verlet_steps(make_params(1.0, 0.0, method=DIRECT, precision=F64_EXACT), 1e-6, 5)
    got = ctx.download()
    ref = oracle.vv_run(pos, vel, m, 1.0, 0.0, 1e-6, 5)[:3]
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kind,most", [("plain", 1.3), ("masses", 1.8)])
def test_time(ctx, kind, most):
    """Before: 1.6 times (library operations) and 2.3 times (both forms)."""
    n = 1500

    def seconds(pos, vel, m, eps):
        ctx.upload(pos, vel, m)
        p = make_params(1.0, eps, method=DIRECT, precision=F64_EXACT)
        t = []
        for _ in range(7):
            t0 = time.perf_counter()
            ctx.verlet_steps(p, 1e-12, 100)
            t.append(time.perf_counter() - t0)
        return min(t)

    pos, vel, m = ics.plummer(n, seed=n)
    assert seconds(*bodies(kind, n)) < most * seconds(pos, vel, m, 0.01)
