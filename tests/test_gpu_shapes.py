"""Kernels at the sizes where their tiles, blocks and dispatch rules meet,
against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bodies_dict
from nbody_b200 import MODE_DIRECT_FP64, scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 64, 511, 512, 513, 1025, 4097, 16385, 33000])
def test_exact_potential_at_tile_edges(engine, oracle, n):
    """The pair potential's 512-row tiles and source chunks: sums of n^2 / 2
    FP64 terms in another order, so 1e-11 relative as for the other sizes."""
    b = scenarios.plummer(n, seed=n)
    b.active[3::7] = 0
    engine.set_state(b)
    d, w = engine.diagnostics(1e-4, pe_mode=0), oracle.energy(bodies_dict(b), 1e-4)
    for k in ("ke", "pe", "e", "lx", "comx", "m"):
        assert d[k] == pytest.approx(w[k], rel=1e-11, abs=1e-14), k


@pytest.mark.parametrize("n", [1, 2, 127, 129, 296, 297, 592, 593, 1184, 1185, 2500])
def test_fp64_direct_at_dispatch_edges(engine, oracle, n):
    """Every block shape of the FP64 sum, and both parities of the step run's
    position buffers: bit for bit the CPU backend's forces and trajectory."""
    b = scenarios.plummer(n, seed=n)
    b.active[5::11] = 0
    want = oracle.direct_forces(b.px, b.py, b.pz, b.mass, b.active, 1e-4)
    got = engine.compute_forces(b.px, b.py, b.pz, b.mass, b.active, 1e-4, MODE_DIRECT_FP64)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)
    for steps in (1, 2, 5):
        engine.set_state(b)
        engine.step(steps, 1e-3, 1e-4, MODE_DIRECT_FP64)
        s, _ = engine.get_state()
        v = oracle.verlet_direct(bodies_dict(b), 1e-4, 1e-3, steps)
        for k in ("px", "py", "pz", "vx", "vy", "vz", "ax", "ay", "az"):
            np.testing.assert_array_equal(getattr(s, k), v[k], err_msg=k)
