"""The segmented reference-form centre of mass of cells of many bodies:
masses and centres of mass of every cell bit-identical to the oracle's serial
insertion, at chain lengths around the segment (256 and 512 bodies at these
sizes) and the single-thread limit, and where the speculation has to fall
back: spatially sorted bodies (the mean drifts), cells around the origin,
planes (one coordinate 0), masses over many binades, massless and negative
bodies."""
import numpy as np
import pytest

import oracle
import physgpu.ics as ics
from physgpu import BARNES_HUT, F64_EXACT, make_params

pytestmark = pytest.mark.gpu


def check(ctx, pos, m):
    ctx.upload(pos, None, m)
    g = ctx.bh_export(make_params(1.0, 0.01, 0.5, BARNES_HUT, F64_EXACT))
    o = oracle.bh_export(pos, m)
    assert np.array_equal(g["count"], o["count"])
    assert np.array_equal(g["mass"], o["mass"])
    assert np.array_equal(g["com"], o["com"])


@pytest.mark.parametrize("n", [255, 511, 512, 513, 767, 768, 1025, 4097, 70000, 140001])
def test_lengths(ctx, n):
    pos, _, _ = ics.plummer(n, seed=n)
    m = np.random.default_rng(n).uniform(0.1, 1.0, n)
    check(ctx, pos, m)


@pytest.mark.parametrize("kind", ["sorted", "centred", "plane", "binades", "massless", "first",
                                  "negative", "equal", "offset"])
def test_fallbacks(ctx, kind):
    rng = np.random.default_rng(5)
    n = 30000
    pos, _, m = ics.plummer(n, seed=3)
    if kind == "sorted":
        pos = pos[np.argsort(pos[:, 0])]
        m = rng.uniform(0.5, 1.5, n)
    elif kind == "centred":  # centres of mass next to 0
        pos = np.concatenate([pos, -pos])
        m = np.ones(2 * n)
    elif kind == "plane":
        pos[:, 2] = 0.0
    elif kind == "binades":
        m = 10.0 ** rng.uniform(-12, 12, n)
    elif kind == "massless":
        m[::3] = 0.0
    elif kind == "first":  # the running mass stays 0 for whole segments
        m[:2000] = 0.0
    elif kind == "negative":
        m = rng.choice([-1.0, 1.0], n, p=[0.2, 0.8])
    elif kind == "equal":
        m[:] = 0.1
    else:
        pos += [1e6, -1e3, 0.0]
    check(ctx, pos, m)
