"""The exact walk with masses of both signs: centres of mass outside their
cells, outside the root cube and beyond the range of the branch-free weight,
bit-identical to the oracle; and not slower for the sign alone."""
import numpy as np
import pytest

import oracle
import physgpu.ics as ics
from physgpu import BARNES_HUT, F64_EXACT, make_params

pytestmark = pytest.mark.gpu


def masses(kind, n):
    rng = np.random.default_rng(n)
    if kind == "signs":
        return rng.choice([-1.0, 1.0], n, p=[0.3, 0.7])
    if kind == "pairs":  # sums of an ulp: centres of mass 2^53 cells away
        return np.resize([1.0, -(1.0 - 2.0 ** -53)], n)
    # sums of an ulp of an ulp: centres of mass beyond 2^98
    e = 2.0 ** -53
    return rng.permutation(np.resize([1.0, -(1.0 - e), -e * (1.0 - e), 0.5], n))


@pytest.mark.parametrize("kind", ["signs", "pairs", "chains"])
@pytest.mark.parametrize("n", [150, 4000, 132_000])
def test_bits(ctx, kind, n):
    pos, _, _ = ics.plummer(n, seed=n)
    m = masses(kind, n)
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(make_params(1.0, 0.01, 0.7, BARNES_HUT, F64_EXACT))
    assert np.array_equal(f, oracle.bh_forces(pos, m, 1.0, 0.01, 0.7))


def test_time_per_interaction(ctx):
    """The f64 test and the library's weights for everything took 1.6 times as
    long as masses of one sign."""
    n = 300_000
    pos, _, m = ics.plummer(n, seed=4)

    def ns(mass):
        ctx.upload(pos, None, mass)
        t = []
        for _ in range(5):
            ctx.gravity_forces(make_params(1.0, 0.01, 0.5, BARNES_HUT, F64_EXACT))
            x = ctx.timings()
            t.append(x["walk_ms"] / x["interactions"])
        return min(t)

    assert ns(m * masses("signs", n)) < 1.35 * ns(m)
