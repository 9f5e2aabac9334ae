"""The branch-free weight's range: separations and softenings next to its upper
and lower limits, on either side, bit-identical in the exact direct sum and
walk."""
import numpy as np
import pytest

import oracle
from physgpu import BARNES_HUT, DIRECT, F64_EXACT, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [98.0, 98.4, 98.6, 99.4, 99.6, -99.9, -100.0, -100.1])
@pytest.mark.parametrize("n", [9, 1300])
def test_limits(ctx, n, exponent):
    rng = np.random.default_rng(n)
    eps = 2.0 ** exponent
    size = 2.0 ** 98 * (1.0 - 2.0 ** -50) if exponent > 0 else 2.0 ** -98
    pos = rng.uniform(-1.0, 1.0, (n, 3)) * size
    pos[0], pos[1] = size, -size  # the largest separation
    pos[2:5] = 2.0 ** -99 if exponent < 0 else size / 2  # and none
    m = rng.uniform(0.5, 2.0, n)
    m[5], m[6] = 2.0 ** 249, 2.0 ** -249
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(make_params(1.0, eps, method=DIRECT, precision=F64_EXACT))
    assert np.array_equal(f, oracle.direct_forces(pos, m, 1.0, eps))
    m[5], m[6] = 2.0 ** 220, 2.0 ** -190
    for half in (1.0, 0.4):  # the root cube on either side of the walk's limit
        ctx.upload(pos * half, None, m)
        f = ctx.gravity_forces(make_params(1.0, eps, 0.5, BARNES_HUT, F64_EXACT))
        assert np.array_equal(f, oracle.bh_forces(pos * half, m, 1.0, eps, 0.5))
