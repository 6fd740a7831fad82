"""The reference-semantics walk where many bodies share one level-21 cell: every
body of such a bucket is summed on its own, so these scenes, in which no cell
is accepted, equal the FP64 direct sum up to rounding."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_err
from nbody_b200 import MODE_BARNES_HUT_REF, MODE_DIRECT_FP64, scenarios
from nbody_b200 import _native as N

pytestmark = pytest.mark.gpu


def _clusters(sizes):
    """Bodies at the corners of a cube, sizes[k] of them at corner k within far
    less than a level-21 cell of it (but not at one point)."""
    b = scenarios.plummer(sum(sizes), seed=len(sizes))
    rng = np.random.default_rng(sum(sizes))
    corner = np.repeat(np.arange(len(sizes)), sizes)
    for k, f in enumerate(("px", "py", "pz")):
        setattr(b, f, ((corner >> k) & 1) * 2.0 - 1.0 + rng.uniform(-1, 1, b.n) * 1e-9)
    b.mass = 1.0 + rng.random(b.n)
    b.radius = np.where(rng.random(b.n) < 0.5, 1e-9, 0.0)
    return b


@pytest.mark.parametrize("shell", [False, True])
@pytest.mark.parametrize("sizes", [[2], [2, 1], [3, 2, 1], [7, 8, 9, 1, 15, 16, 17, 33],
                                   [100, 1, 500, 2, 31, 3, 1, 64], [1, 1000], [1, 1, 1, 1, 2]])
def test_buckets_equal_the_direct_sum(engine, oracle, sizes, shell):
    """Sums of n terms of one sign pattern in another order, FP64: n rounding
    units of the largest term, 1e-12 of the result for these scenes."""
    b = _clusters(sizes)
    if b.n > 20:
        b.active[5::9] = 0
    eps = 1e-3
    want = oracle.direct_forces(b.px, b.py, b.pz, b.mass, b.active, eps, radius=b.radius,
                                shell=shell)
    engine.set_param(N.PARAM_THETA, 0.2)
    got = engine.compute_forces(b.px, b.py, b.pz, b.mass, b.active, eps,
                                MODE_BARNES_HUT_REF | (N.FLAG_SHELL_THEOREM if shell else 0),
                                radius=b.radius)
    engine.set_param(N.PARAM_THETA, 0.5)
    # each body's error in units of the sum of its terms' sizes
    scale = b.mass.sum() * 1e-9 / eps ** 3 + np.sqrt((np.array(want) ** 2).sum(0))
    err = np.sqrt(((np.array(got) - np.array(want)) ** 2).sum(0))
    assert (err <= 1e-12 * scale).all()
    far = b.active == 1
    if len(sizes) > 1 and far.sum() > 1:
        assert rel_err(got, want)[far].max() < 1e-9


def test_a_large_bucket_keeps_every_lane_at_work(engine):
    """One body far away puts the other 20,010 into a single cell: the walk is
    a direct sum then, and its time on the device stays within five times that
    of the FP64 direct sum (ten times with each body's terms on 4 of 32 lanes)."""
    b = scenarios.plummer(20_011, seed=2)
    for k in ("px", "py", "pz"):
        setattr(b, k, getattr(b, k) * 1e-9)
    b.px[0] = 100.0

    def ms(mode):
        t = []
        for _ in range(4):
            engine.compute_forces(b.px, b.py, b.pz, b.mass, b.active, 1e-4, mode)
            t.append(engine.timings()[N.T_TOTAL])
        return min(t)

    assert ms(MODE_BARNES_HUT_REF) < 5.0 * ms(MODE_DIRECT_FP64)
