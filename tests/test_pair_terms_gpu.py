"""Pair-term arithmetic at the edges of its ranges: scales far from one,
overflowing squares, and the F64 target layouts of the group walk.

Tolerance of the F64 forms: a pair term has fewer than 10 roundings and a
sum of n terms at most n more, each of u = 2^-53 relative to the largest
partial sum; with n <= 200 bodies around a common scale 1e-12 leaves a factor
of 40."""
import numpy as np
import pytest

import oracle
import physgpu.ics as ics
from physgpu import BARNES_HUT, DIRECT, F64, F64_EXACT, GROUP_WALK, make_params

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return np.linalg.norm(a - b, axis=1) / np.maximum(np.linalg.norm(b, axis=1), 1e-300)


@pytest.mark.parametrize("scale", [1e-45, 1e-20, 1.0, 1e11, 1e26, 1e60])
def test_f64_scales(ctx, scale):
    pos, _, m = ics.plummer(150, seed=4)
    pos = pos * scale
    ctx.upload(pos, None, m)
    ref = oracle.direct_forces(pos, m, 1.0, 0.0)
    for p in (make_params(1.0, 0.0, 0.0, DIRECT, F64),
              make_params(1.0, 0.0, 0.0, BARNES_HUT, F64),
              make_params(1.0, 0.0, 0.0, BARNES_HUT, F64, 8, GROUP_WALK)):
        if scale < 1e-8 and p.method == BARNES_HUT:
            continue  # closer than the guard cell: the tree stores one body of it
        assert rel_err(ctx.gravity_forces(p), ref).max() < 1e-12


def test_f64_overflowed_square_adds_nothing(ctx):
    """|r|^2 beyond the f64 range: the reference's term is r * (x / inf) = 0."""
    pos = np.array([[0.0, 0, 0], [1.0, 0.5, 0.25], [1e200, 0, 0]])
    m = np.array([1.0, 2.0, 3.0])
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(make_params(1.0, 0.01, precision=F64))
    ref = oracle.direct_forces(pos, m, 1.0, 0.01)
    assert np.all(f[2] == 0.0) and np.all(ref[2] == 0.0)
    assert rel_err(f[:2], ref[:2]).max() < 1e-12


@pytest.mark.parametrize("n", [8, 9, 31, 32, 33, 40, 41, 48, 49, 64])
def test_f64_group_layouts(ctx, n):
    """A group of n bodies beside 70 far ones (a list of 70, padded to 72): every
    target layout of the F64 evaluation, in-group and list passes, against
    the direct sum at theta = 0."""
    pos, _, m = ics.plummer(n, seed=200 + n)
    far = np.array([500.0, 300.0, 400.0]) + np.random.default_rng(n).normal(size=(70, 3))
    pos = np.concatenate([pos, far])
    m = np.concatenate([m, np.full(70, 0.5)])
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(make_params(1.0, 0.01, 0.0, BARNES_HUT, F64, 1, GROUP_WALK))
    assert ctx.timings()["interactions"] == (n + 70) * (n + 69)
    assert rel_err(f, oracle.direct_forces(pos, m, 1.0, 0.01)).max() < 1e-12


@pytest.mark.parametrize("n", [2, 7, 8, 9, 33, 1183, 1184, 1185, 1301])
@pytest.mark.parametrize("eps", [0.0, 0.01])
def test_exact_direct_blocks_and_ranges(ctx, n, eps):
    """Bit-identical at the edges of the target blocks (8 targets up to 1184
    bodies, 10 beyond), with sources and targets whose masses or coordinates
    leave the range of the branch-free weight, massless bodies, and without
    softening."""
    pos, _, m = ics.plummer(n, seed=n)
    m[::5] *= 1e-120
    m[1::7] = 0.0
    pos[n // 2] *= 1e35
    if n > 30:
        pos[3] *= 1e-40 if eps else 1.0
        m[17] *= 1e200
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(make_params(1.0, eps, method=DIRECT, precision=F64_EXACT))
    assert np.array_equal(f, oracle.direct_forces(pos, m, 1.0, eps))


@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("n", [9, 130, 1190])
def test_exact_fused_ticks(ctx, n, steps):
    """Runs of ticks with one kernel per pair-wise tick equal the reference's
    tick loop bit for bit whatever the number of ticks, state and all."""
    pos, vel, m = ics.plummer(n, seed=n + 1)
    ctx.upload(pos, vel, m)
    p = make_params(1.0, 0.05, method=DIRECT, precision=F64_EXACT)
    ctx.verlet_steps(p, 1e-3, steps)
    x, v, a = ctx.download()
    xr, vr, ar = oracle.vv_run(pos, vel, m, 1.0, 0.05, 1e-3, steps)[:3]
    assert np.array_equal(x, xr) and np.array_equal(v, vr) and np.array_equal(a, ar)
