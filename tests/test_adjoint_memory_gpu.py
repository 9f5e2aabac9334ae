"""The gradient where the device has no room for the positions of every step:
the caller's checkpoint interval is used, with the same results bit for bit."""
import numpy as np
import pytest

import physgpu
import physgpu.ics as ics
from physgpu import DIRECT, F64, make_params

pytestmark = pytest.mark.gpu


def test_interval_when_memory_is_short():
    torch = pytest.importorskip("torch")
    n, steps = 20_000, 500  # 240 MB of positions; 100 MB with an interval of 25
    pos, vel, m = ics.plummer(n, seed=4)
    p = make_params(1.0, 0.05, method=DIRECT, precision=F64)
    with physgpu.Context(0) as ctx:
        ctx.upload(pos, vel, m)
        ref = ctx.adjoint(p, 1e-4, steps, pos, checkpoint=25)
    with physgpu.Context(0) as ctx:
        ctx.upload(pos, vel, m)
        free = torch.cuda.mem_get_info(0)[0]
        taken = torch.empty(free - (160 << 20), dtype=torch.uint8, device="cuda")
        try:
            got = ctx.adjoint(p, 1e-4, steps, pos, checkpoint=25)
        finally:
            del taken
            torch.cuda.empty_cache()
    for a, b in zip(ref, got):
        assert np.array_equal(a, b)
