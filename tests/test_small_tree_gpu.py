"""Bodies and cells of small trees are put in order by counting (one kernel)
up to 12288 bodies and 6144 cells: the order at the edges of the tiles and of
the ranges, with whole runs of equal keys, and a group walk over the order."""
import numpy as np
import pytest

import physgpu.ics as ics
from physgpu import BARNES_HUT, DIRECT, F64, GROUP_WALK, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 33, 1023, 1024, 1025, 12287, 12288, 12289])
@pytest.mark.parametrize("kind", ["spread", "clumps"])
def test_order(ctx, n, kind):
    pos, _, m = ics.plummer(n, seed=n)
    if kind == "clumps":  # equal keys (index decides) and keys that differ in the low word only
        rng = np.random.default_rng(n)
        pos[n // 3:n // 2] = pos[n // 3]
        k = n - n // 4
        pos[k:] = pos[n // 2] + rng.normal(scale=1e-8, size=(n - k, 3))
    ctx.upload(pos, None, m)
    g = ctx.bh_export(make_params(1.0, 0.01, 0.5, BARNES_HUT, F64))
    assert np.array_equal(g["perm"], np.lexsort((np.arange(n), g["keys_lo"], g["keys_hi"])))


@pytest.mark.parametrize("n", [5000, 13800, 14400, 15000])  # cells on both sides of 6144
def test_walk_over_order(ctx, n):
    """theta 0 opens every cell: each pair once, whatever the order of the sum."""
    pos, _, m = ics.plummer(n, seed=3)
    ctx.upload(pos, None, m)
    p = make_params(1.0, 0.02, 0.0, BARNES_HUT, F64, leaf_cap=8, flags=GROUP_WALK)
    got = ctx.gravity_accel(p)
    ref = ctx.gravity_accel(make_params(1.0, 0.02, 0.0, DIRECT, F64))
    # both sums: n terms of at most 1 / eps^2 * m in size, each within a few
    # units in the last place, added in some order
    size = np.zeros(n)
    for k in range(0, n, 500):
        d2 = ((pos[k:k + 500, None] - pos[None]) ** 2).sum(-1) + 0.02 ** 2
        size[k:k + 500] = (m[None] / d2).sum(-1)
    bound = 2 * (n + 16) * 2.0 ** -53 * size
    assert (np.abs(got - ref).max(-1) <= bound).all()
