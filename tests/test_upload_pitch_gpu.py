"""Uploads of few bodies into a context that once held very many: its arrays
lie 2^31 bytes apart, more than one strided copy may span."""
import numpy as np
import pytest

import oracle
import physgpu
import physgpu.ics as ics
from physgpu import DIRECT, F64_EXACT, make_params

pytestmark = pytest.mark.gpu


def test_small_uploads_after_a_large_one():
    n = 1 << 28
    with physgpu.Context(0) as ctx:
        one = np.zeros(n)  # 34 GB of state on the device from one host array
        st = ctx.lib.phys_state_upload(ctx.h, n, *[physgpu._p(one)] * 3, None, None, None,
                                       physgpu._p(one))
        del one
        if st == physgpu.ERR_OOM:
            pytest.skip("device memory taken")
        assert st == physgpu.OK
        pos, vel, m = ics.plummer(500, seed=1)
        ref = oracle.direct_forces(pos, m, 1.0, 0.01)
        p = make_params(1.0, 0.01, method=DIRECT, precision=F64_EXACT)
        ctx.upload(pos, vel, m)
        assert np.array_equal(ctx.gravity_forces(p), ref)
        x, v, a = ctx.download()
        assert np.array_equal(x, pos) and np.array_equal(v, vel) and not a.any()
        ctx.upload_sectors(np.zeros((500, 3), np.int64), pos, 1e12, m)
        assert np.array_equal(ctx.gravity_forces(p), ref)
