"""The exact walk's scratch follows the tasks that the tree has; a tree of
more tasks than there is room for is walked as one."""
import numpy as np
import pytest

import oracle
import physgpu
import physgpu.ics as ics
from physgpu import BARNES_HUT, F64_EXACT, make_params

pytestmark = pytest.mark.gpu

P = make_params(1.0, 0.01, 0.6, BARNES_HUT, F64_EXACT)


def cusp(n):
    """Nested cells with much of the mass each: radii over 22 binades."""
    rng = np.random.default_rng(n)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    return 10.0 * 2.0 ** -rng.uniform(0, 22, n)[:, None] * u, np.full(n, 1.0 / n)


def test_held_memory():
    torch = pytest.importorskip("torch")
    pos, _, m = ics.plummer(10_000, seed=1)
    with physgpu.Context(0) as ctx:
        ctx.upload(pos[:50], None, m[:50])
        ctx.gravity_forces(P)  # kernels loaded
        free = torch.cuda.mem_get_info(0)[0]
        ctx.upload(pos, None, m)
        f = ctx.gravity_forces(P)
        held = free - torch.cuda.mem_get_info(0)[0]
    assert np.array_equal(f, oracle.bh_forces(pos, m, 1.0, 0.01, 0.6))
    assert held < 80e6  # 24 bytes a task and target: about 100 tasks


@pytest.mark.parametrize("n", [40, 3000, 20_000, 36_000, 70_000, 120_000])
def test_nested_cells(ctx, n):
    pos, m = cusp(n)
    ctx.upload(pos, None, m)
    assert np.array_equal(ctx.gravity_forces(P), oracle.bh_forces(pos, m, 1.0, 0.01, 0.6))
