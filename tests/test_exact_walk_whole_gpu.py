"""The exact walk of more than 131 072 targets: deep chains with the cells of
several depths waiting, pairs without softening and massless cells,
bit-identical to the oracle's recursive walk; and shares of the targets that
start anywhere, on the split walk, on this one, and with none left."""
import numpy as np
import pytest
import torch

import oracle
import physgpu
import physgpu.ics as ics
from physgpu import BARNES_HUT, F64_EXACT, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,theta", [("clumps", 1.1), ("unsoftened", 0.9), ("massless", 0.6),
                                        ("tiny", 0.7)])
def test_ranges(ctx, kind, theta):
    n = 131_200
    rng = np.random.default_rng(5)
    pos, _, m = ics.plummer(n, seed=8)
    eps = 0.02
    if kind == "clumps":  # coincident bodies and a clump down to the guard depth
        pos[200:230] = pos[200]
        pos[900:1100] = pos[900] + rng.normal(scale=1e-7, size=(200, 3))
    elif kind == "unsoftened":
        eps = 0.0
    elif kind == "massless":
        m[pos[:, 0] > 0.3] = 0.0
    else:  # the library's weights
        m *= 1e-90
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(make_params(1.0, eps, theta, BARNES_HUT, F64_EXACT))
    assert np.array_equal(f, oracle.bh_forces(pos, m, 1.0, eps, theta))


@pytest.mark.parametrize("n,world", [(264_000, 2), (264_000, 5), (700, 3), (300, 8)])
def test_shares(ctx, n, world):
    pos, _, m = ics.plummer(n, seed=3)
    p = make_params(1.0, 0.02, 0.9, BARNES_HUT, F64_EXACT)
    ctx.upload(pos, None, m)
    c = physgpu.share_chunk(n, world)
    blocks = [torch.empty(3 * c, dtype=torch.float64, device="cuda") for _ in range(world)]
    for r in range(world):
        ctx.gravity_accel_share(p, r, world, blocks[r].data_ptr())
    gathered = torch.cat(blocks)
    ctx.gravity_accel_unshare(world, gathered.data_ptr())
    torch.cuda.synchronize()
    _, _, a = ctx.download()
    assert np.array_equal(a, oracle.accel(oracle.bh_forces(pos, m, 1.0, 0.02, 0.9), m))
