"""F32C ensemble with the state in registers (32 lanes, lanes by size) against
the state in shared memory (a fixed 16 lanes): for up to 16 bodies both add the
same terms in the same order, so the results are the same bits."""
import numpy as np
import pytest

import physgpu
from physgpu import F32C, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config", [32, physgpu.ENS_BY_SIZE,
                                    physgpu.ENS_BY_SIZE | physgpu.ens_warps(4)])
@pytest.mark.parametrize("eps", [0.0, 1e-2])
@pytest.mark.parametrize("nsys", [1, 40, 2400])  # one warp, a partial chip, every warp and more
def test_registers_equal_shared(ctx, nsys, eps, config):
    rng = np.random.default_rng(nsys)
    sizes = np.resize([16, 1, 9, 2, 8, 3, 15, 4, 7], nsys)
    off = np.concatenate([[0], np.cumsum(sizes)])
    n = int(off[-1])
    pos = rng.uniform(-1, 1, (n, 3))
    vel = rng.normal(0, 0.3, (n, 3))
    m = np.exp(rng.uniform(np.log(0.1), np.log(10), n))
    out = []
    for group in (16, config):
        ctx.ensemble_load(off, pos, vel, m)
        for steps, chunk in ((3, 0), (4, 2)):  # first with the accelerations to form
            ctx.ensemble_run(make_params(1.0, eps, precision=F32C), 1e-4, steps, group=group,
                             chunk=chunk)
        out.append(ctx.ensemble_download())
    for a, b in zip(*out):
        assert np.array_equal(a, b)
