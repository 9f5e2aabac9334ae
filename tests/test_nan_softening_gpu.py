"""A NaN softening makes every pair term NaN: each F64 entry point reports it
as a non-finite result, as the exact and the F32C forms do, instead of
returning zeros."""
import ctypes
import math

import numpy as np
import pytest

import physgpu
import physgpu.ics as ics
from physgpu import BARNES_HUT, DIRECT, F32C, F64, F64_EXACT, GROUP_WALK, PhysError, make_params

pytestmark = pytest.mark.gpu

FORMS = [(DIRECT, F64, 1, 0), (BARNES_HUT, F64, 1, 0), (BARNES_HUT, F64, 8, 0),
         (BARNES_HUT, F64, 8, GROUP_WALK), (DIRECT, F64_EXACT, 1, 0),
         (BARNES_HUT, F64_EXACT, 1, 0), (DIRECT, F32C, 1, 0), (BARNES_HUT, F32C, 8, GROUP_WALK)]


@pytest.mark.parametrize("n", [2, 41, 700])
@pytest.mark.parametrize("form", FORMS)
def test_gravity(ctx, form, n):
    method, precision, leaf_cap, flags = form
    pos, vel, m = ics.plummer(n, seed=n)
    ctx.upload(pos, vel, m)
    p = make_params(1.0, math.nan, 0.5, method, precision, leaf_cap, flags)
    for call in (lambda: ctx.gravity_accel(p), lambda: ctx.gravity_forces(p),
                 lambda: ctx.verlet_steps(p, 1e-3, 2)):
        with pytest.raises(PhysError) as e:
            call()
        assert e.value.status == physgpu.ERR_NONFINITE
        ctx.upload(pos, vel, m)


def test_targets_and_trajectories(ctx):
    pos, vel, m = ics.plummer(300, seed=2)
    ctx.upload(pos, vel, m)
    p = make_params(1.0, math.nan, 0.5, DIRECT, F64)
    for call in (lambda: ctx.direct_accel_targets(p, np.arange(7)),
                 lambda: ctx.trajectory_loss(p, 1e-3, 2, pos),
                 lambda: ctx.adjoint(p, 1e-3, 2, pos)):
        with pytest.raises(PhysError) as e:
            call()
        assert e.value.status == physgpu.ERR_NONFINITE


def test_noalloc():
    torch = pytest.importorskip("torch")
    lib = physgpu.load_library()
    pos, _, m = ics.plummer(300, seed=2)
    X = [torch.from_numpy(np.ascontiguousarray(c)).cuda() for c in (*pos.T, m)]
    A = [torch.zeros(300, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    err = ctypes.create_string_buffer(256)
    st = lib.phys_direct_accel_noalloc(300, *[t.data_ptr() for t in X], 1.0, math.nan, F64,
                                       *[t.data_ptr() for t in A], None, err, 256)
    assert st == physgpu.ERR_NONFINITE
