"""The exact Barnes-Hut walk split over subtrees (up to 131 072 targets) and
the one walk per target beyond: bit-identical to the oracle's recursive walk
at the edges of the split, for trees without upper cells, deep chains, masses
that rule out the f32 opening test or the branch-free weight, and shares."""
import numpy as np
import pytest

import oracle
import physgpu.ics as ics
from physgpu import BARNES_HUT, F64_EXACT, make_params

pytestmark = pytest.mark.gpu


def exact(theta=0.5, eps=0.01, G=1.0):
    return make_params(G, eps, theta, BARNES_HUT, F64_EXACT)


@pytest.mark.parametrize("theta", [0.0, 0.5, 1.2])
@pytest.mark.parametrize("n", [2, 3, 7, 8, 9, 31, 32, 33, 64, 129, 1500])
def test_small(ctx, n, theta):
    pos, _, m = ics.plummer(n, seed=n)
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(exact(theta))
    assert np.array_equal(f, oracle.bh_forces(pos, m, 1.0, 0.01, theta))


@pytest.mark.parametrize("n", [8192, 65536, 65537])
def test_split_edges(ctx, n):
    pos, _, m = ics.galaxy(n, seed=n)
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(exact(0.6, 0.02))
    assert np.array_equal(f, oracle.bh_forces(pos, m, 1.0, 0.02, 0.6))


@pytest.mark.parametrize("kind", ["unsoftened", "zero", "negative", "tiny", "far", "clumps"])
def test_ranges(ctx, kind):
    rng = np.random.default_rng(11)
    pos, _, m = ics.plummer(2500, seed=6)
    eps = 0.01
    if kind == "unsoftened":
        eps = 0.0
    elif kind == "zero":  # massless bodies and cells (gated, gravity_tree.rs:201)
        m[pos[:, 0] > 0.3] = 0.0
    elif kind == "negative":  # centres of mass outside their cells
        m *= rng.choice([-1.0, 1.0], len(m), p=[0.3, 0.7])
    elif kind == "tiny":
        m *= 1e-90
    elif kind == "far":
        pos[7] = [3e33, -2e33, 1e33]
    else:  # deep chains: coincident bodies and a clump at the guard depth
        pos[100:160] = pos[100]
        pos[300:420] = pos[300] + rng.normal(scale=1e-9, size=(120, 3))
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(exact(0.5, eps))
    assert np.array_equal(f, oracle.bh_forces(pos, m, 1.0, eps, 0.5))


@pytest.mark.parametrize("kind,theta", [("negative", 0.7), ("clumps", 1.1), ("unsoftened", 0.9)])
def test_many_targets_ranges(ctx, kind, theta):
    """Many targets: the f64 test for every cell, deep chains
    with the cells of several depths waiting, and the library's weights."""
    n = 65_700
    rng = np.random.default_rng(5)
    pos, _, m = ics.plummer(n, seed=8)
    eps = 0.02
    if kind == "negative":
        m *= rng.choice([-1.0, 1.0], n, p=[0.3, 0.7])
    elif kind == "clumps":
        pos[200:230] = pos[200]
        pos[900:1100] = pos[900] + rng.normal(scale=1e-7, size=(200, 3))
    else:
        eps = 0.0
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(exact(theta, eps))
    assert np.array_equal(f, oracle.bh_forces(pos, m, 1.0, eps, theta))


@pytest.mark.parametrize("n,ic", [(30_000, "galaxy"), (60_000, "plummer"), (90_000, "plummer"),
                                  (131_072, "galaxy"), (131_073, "plummer")])
def test_task_sizes(ctx, n, ic):
    """One size for each share of the bodies that the tasks are made from, and
    both sides of the last split."""
    pos, _, m = getattr(ics, ic)(n, seed=2)
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(exact(0.6, 0.02))
    assert np.array_equal(f, oracle.bh_forces(pos, m, 1.0, 0.02, 0.6))


def test_whole_walk_far_masses(ctx):
    """Beyond the split: masses of both signs and unsoftened pairs."""
    n = 131_500
    pos, _, m = ics.plummer(n, seed=8)
    m *= np.random.default_rng(5).choice([-1.0, 1.0], n, p=[0.3, 0.7])
    ctx.upload(pos, None, m)
    f = ctx.gravity_forces(exact(0.8, 0.0))
    assert np.array_equal(f, oracle.bh_forces(pos, m, 1.0, 0.0, 0.8))
