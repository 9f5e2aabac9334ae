"""The F32C ensemble runs on more warps an SM from three systems a warp on: a
system's trajectory is the same bits on either side of that number."""
import numpy as np
import pytest

from physgpu import DIRECT, F32C, ENS_BY_SIZE, ens_warps, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config", [32, ENS_BY_SIZE])
@pytest.mark.parametrize("warps", [2, 4])
def test_few_and_many_systems(ctx, config, warps):
    rng = np.random.default_rng(warps)
    sizes = rng.integers(2, 65, 7300)  # 3 x 16 x 148 = 7104
    off = np.concatenate([[0], np.cumsum(sizes)])
    pos, vel = rng.normal(size=(off[-1], 3)), 0.1 * rng.normal(size=(off[-1], 3))
    m = rng.uniform(0.1, 1.0, off[-1])
    p = make_params(1.0, 0.01, method=DIRECT, precision=F32C)

    def run(systems):
        n = off[systems]
        ctx.ensemble_load(off[:systems + 1], pos[:n], vel[:n], m[:n])
        ctx.ensemble_run(p, 1e-3, 20, config | ens_warps(warps))
        return ctx.ensemble_download()

    few, many = run(300), run(7300)
    for a, b in zip(few, many):
        assert np.array_equal(a, b[:off[300]])
