"""Centre-of-mass segments whose speculation leaves the range of the fast
division: bit-identical cells, and the time of the segments, not of one serial
chain, where the true values stay in range."""
import numpy as np
import pytest

import oracle
import physgpu.ics as ics
from physgpu import BARNES_HUT, F64_EXACT, make_params

pytestmark = pytest.mark.gpu


def bodies(kind, n):
    rng = np.random.default_rng(n)
    pos, _, m = ics.plummer(n, seed=n)
    if kind == "plane":
        pos[:, 2] = 0.0
        m[:] = 1.0
    elif kind == "line":
        pos[:, 1:] = 0.0
        m = rng.uniform(0.5, 1.5, n)
    elif kind == "signs":  # running masses positive but for the first few
        m = rng.choice([-1.0, 1.0], n, p=[0.3, 0.7])
    elif kind == "cancelling":  # running masses around 0 all along
        m = np.resize([1.0, -1.0, 0.75, -0.75], n) * rng.uniform(0.9, 1.1, n)
    elif kind == "negative":
        m = -m
    elif kind == "massless":  # a whole cell's worth, then some
        m[:n // 3] = 0.0
    elif kind == "heavy":  # running masses beyond the range from the middle on
        m[n // 2] = 1e200
    elif kind == "small":  # a coordinate below the range
        pos[:, 1] *= 1e-160
    elif kind == "flat half":  # the centre of mass leaves 0 in mid-chain
        pos[:n // 2, 2] = 0.0
    return pos, m


@pytest.mark.parametrize("kind", ["plane", "line", "signs", "cancelling", "negative", "massless",
                                  "heavy", "small", "flat half"])
@pytest.mark.parametrize("n", [1100, 30000, 140001])
def test_bits(ctx, kind, n):
    check(ctx, *bodies(kind, n))


@pytest.mark.parametrize("kind", ["plane", "signs", "massless", "flat half"])
def test_bits_refined(ctx, kind):  # longest chains: windows moved and run again
    check(ctx, *bodies(kind, 510_000))


def check(ctx, pos, m):
    ctx.upload(pos, None, m)
    g = ctx.bh_export(make_params(1.0, 0.01, 0.5, BARNES_HUT, F64_EXACT))
    o = oracle.bh_export(pos, m)
    assert np.array_equal(g["count"], o["count"])
    assert np.array_equal(g["mass"], o["mass"])
    assert np.array_equal(g["com"], o["com"])


@pytest.mark.parametrize("kind", ["plane", "massless"])
def test_no_serial_fallback(ctx, kind):
    """Whole cells on one serial chain took 9 to 14 times as long."""
    n = 100_000

    def tree_ms(pos, m):
        ctx.upload(pos, None, m)
        t = []
        for _ in range(5):
            ctx.gravity_forces(make_params(1.0, 0.01, 0.5, BARNES_HUT, F64_EXACT))
            t.append(ctx.timings()["tree_ms"])
        return min(t)

    assert tree_ms(*bodies(kind, n)) < 4.0 * tree_ms(*bodies("plain", n))
