"""Kernels at the sizes where their tiles, blocks and dispatch rules meet,
against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bodies_dict
from helpers import rel_err
from nbody_b200 import (MODE_BARNES_HUT, MODE_BARNES_HUT_REF, MODE_DIRECT, MODE_DIRECT_FP64,
                        scenarios)
from nbody_b200 import _native as N

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


def _nested_corner(levels=9):
    """A cell whose corner octant is subdivided again and again, every other
    octant of each level holding one body in each of its own octants: a walk
    that opens everything leaves 56 nodes behind on each level."""
    pts = [(0.0005,) * 3, (0.9995,) * 3]
    for lev in range(levels):
        for o in range(1, 8):
            for q in range(8):
                pts.append(tuple(2.0 ** -(lev + 1) * (((o >> a) & 1) + 0.25 + 0.5 * ((q >> a) & 1))
                                 for a in range(3)))
    p = np.array(pts) * 2.002 - 1.001  # the octree's cube of a [-1, 1] box
    n = len(p)
    b = scenarios.plummer(n, seed=7)
    b.px, b.py, b.pz = (np.ascontiguousarray(p[:, k]) for k in range(3))
    b.mass = 1.0 + np.arange(n) % 5
    return b


@pytest.mark.parametrize("scene", [1, 2, 3, 4, 5, 31, 33, 1000, "corner", "disk"])
def test_reference_walk_at_group_edges(engine, oracle, scene):
    """The four-body warps of the reference walk, its narrow rounds when the
    stack fills (the nested corner) and its shell leaves, against the oracle's
    walk: the same cells, so FP64 rounding apart (the mode's 1e-9)."""
    shell, theta = scene == "disk", 0.2 if scene == "corner" else 0.5
    if shell:
        b = scenarios.collisional_disk(601, seed=9, radius_scale=3000.0)
    else:
        b = _nested_corner() if scene == "corner" else scenarios.plummer(scene, seed=scene)
    if b.n > 4:
        b.active[4::13] = 0
    want = oracle.bh_forces(b.px, b.py, b.pz, b.mass, b.active, 1e-4, theta, radius=b.radius,
                            shell=shell)
    engine.set_param(N.PARAM_THETA, theta)
    got = engine.compute_forces(b.px, b.py, b.pz, b.mass, b.active, 1e-4,
                                MODE_BARNES_HUT_REF | (N.FLAG_SHELL_THEOREM if shell else 0),
                                radius=b.radius)
    engine.set_param(N.PARAM_THETA, 0.5)
    if b.n == 1:
        assert got[0][0] == got[1][0] == got[2][0] == 0.0
        return
    assert rel_err(got, want)[b.active == 1].max() < 1e-9


@pytest.mark.parametrize("shell", [False, True])
@pytest.mark.parametrize("eps", [0.0, 1e-4])
@pytest.mark.parametrize("n", [1, 33, 65, 1000, 20011, 500000])
def test_group_walk_helping_range(engine, oracle, n, eps, shell):
    """The walk with and without helping warps (n on both sides of the rule),
    64- and 32-body groups, with zero softening too: the sampled bodies within
    the mode's 1e-3 rms of the FP64 direct sum, the counts of a second call the
    same and its forces the same bits."""
    b = scenarios.plummer(n, seed=n)
    b.radius[:] = 1e-3
    flags = MODE_BARNES_HUT | (N.FLAG_SHELL_THEOREM if shell else 0)
    engine.set_param(N.PARAM_THETA, 0.5)

    def forces():
        f = engine.compute_forces(b.px, b.py, b.pz, b.mass, b.active, eps, flags, radius=b.radius)
        return np.array(f), engine.counters()[:2].tolist()

    got, counts = forces()
    again, counts2 = forces()
    np.testing.assert_array_equal(got, again)
    assert counts == counts2
    t = np.unique(np.linspace(0, n - 1, min(n, 256)).astype(np.int32))
    want = np.array(oracle.direct_forces_targets(b.px, b.py, b.pz, b.mass, b.active, eps, t,
                                                 radius=b.radius, shell=shell))
    den = np.sqrt((want ** 2).sum(0))
    err = np.sqrt(((got[:, t] - want) ** 2).sum(0))[den > 0] / den[den > 0]
    assert np.isfinite(got).all()
    assert err.size == 0 or np.sqrt(np.mean(err ** 2)) < 1e-3


@pytest.mark.parametrize("n", [1, 1000, 2016, 2017, 6001, 30000, 300001])
def test_state_round_trip_at_transfer_sizes(engine, n):
    """Host arrays below and above the pinned half and the pool's chunks, rows
    that are views, and flags: every array comes back bit for bit."""
    rng = np.random.default_rng(n)
    b = scenarios.plummer(n, seed=n)
    for k in ("px", "vy", "az", "radius"):
        setattr(b, k, rng.standard_normal(2 * n)[::2])  # not contiguous
    for k in ("ax", "ay"):
        setattr(b, k, rng.standard_normal(n))
    b.active = rng.integers(0, 2, n).astype(np.uint8)
    engine.set_state(b)
    s, ids = engine.get_state()
    for k in ("px", "py", "pz", "vx", "vy", "vz", "ax", "ay", "az", "mass", "radius", "active"):
        np.testing.assert_array_equal(getattr(s, k), getattr(b, k), err_msg=k)
    np.testing.assert_array_equal(ids, np.arange(n))


@pytest.mark.parametrize("n", [30000, 120001, 300001])
@pytest.mark.parametrize("fields", ["px py pz mass", "px py pz vx vy vz mass radius ax ay az", "vz"])
def test_state_round_trip_from_pinned_arrays(engine, n, fields):
    """Pinned arrays among pageable ones, at sizes that go by the pool: every
    array comes back bit for bit."""
    import torch

    rng = np.random.default_rng(n)
    b = scenarios.plummer(n, seed=n)
    for k in ("ax", "ay", "az"):
        setattr(b, k, rng.standard_normal(n))
    keep = {k: torch.from_numpy(np.ascontiguousarray(getattr(b, k))).pin_memory()
            for k in fields.split()}
    for k, t in keep.items():
        setattr(b, k, t.numpy())
    for _ in range(3):
        engine.set_state(b)
        s, _ = engine.get_state()
        for k in ("px", "py", "pz", "vx", "vy", "vz", "ax", "ay", "az", "mass", "radius"):
            np.testing.assert_array_equal(getattr(s, k), getattr(b, k), err_msg=k)


def test_transfers_of_two_threads():
    """Two handles in two threads share the copy pool: each gets its own data."""
    from concurrent.futures import ThreadPoolExecutor

    from nbody_b200 import Engine

    def one(seed):
        b = scenarios.plummer(200_000 + seed, seed=seed)
        with Engine(b.n) as e:
            for _ in range(6):
                e.set_state(b)
                s, _ = e.get_state()
                for k in ("px", "vz", "mass"):
                    np.testing.assert_array_equal(getattr(s, k), getattr(b, k))
        return True

    with ThreadPoolExecutor(2) as ex:
        assert all(ex.map(one, (1, 2)))


@pytest.mark.parametrize("n", [1, 2, 257, 37888, 37889, 303104, 303105, (1 << 20) + 1])
def test_keys_and_tree_at_dispatch_edges(engine, oracle, n):
    """The key kernel's and the node numbering's variants: keys and cube bit
    for bit, the sorted order stable, and nodes that partition the bodies."""
    b = scenarios.plummer(n, seed=3)
    b.active[7::17] = 0
    keys, _, cube = engine.morton_keys(b.px, b.py, b.pz, b.active, 1)
    want, _, want_cube = oracle.morton_cube(b.px, b.py, b.pz, b.active)
    np.testing.assert_array_equal(keys, want)
    np.testing.assert_array_equal(cube, want_cube)
    t = engine.build_octree(b.px, b.py, b.pz, b.mass, b.active, 24)
    order = np.argsort(want, kind="stable")
    np.testing.assert_array_equal(t["sorted_idx"], order)
    na = int(b.active.sum())
    leaf = t["n_children"] == 0
    assert t["body_count"][0] == na and t["body_count"][leaf].sum() == na
    first = np.sort(t["body_first"][leaf])
    np.testing.assert_array_equal(first, np.cumsum(np.r_[0, t["body_count"][leaf][np.argsort(
        t["body_first"][leaf])]])[:-1])
    inner = np.flatnonzero(~leaf)
    m = np.add.reduceat(t["mass"][1:], t["first_child"][inner][np.argsort(
        t["first_child"][inner])] - 1) if inner.size else np.empty(0)
    np.testing.assert_allclose(m, t["mass"][inner][np.argsort(t["first_child"][inner])],
                               rtol=1e-12)


@pytest.mark.parametrize("shell", [False, True])
@pytest.mark.parametrize("n", [1, 2, 255, 257, 1025, 2561, 4097, 12345])
def test_fp32_direct_at_row_and_chunk_edges(engine, oracle, n, shell):
    """Rows of 256 targets, staged 256-source pieces, j-tiles of 1024 and
    chunks that end inside them: the mode's 2e-6 rms (1e-5 with shells)."""
    b = scenarios.collisional_disk(n, seed=n, radius_scale=300.0) if shell and n > 1 else \
        scenarios.plummer(n, seed=n)
    flags = MODE_DIRECT | (N.FLAG_SHELL_THEOREM if shell else 0)
    got = engine.compute_forces(b.px, b.py, b.pz, b.mass, b.active, 1e-3, flags, radius=b.radius)
    want = oracle.direct_forces(b.px, b.py, b.pz, b.mass, b.active, 1e-3, radius=b.radius,
                                shell=shell)
    if b.n == 1:
        assert got[0][0] == got[1][0] == got[2][0] == 0.0
        return
    assert np.sqrt(np.mean(rel_err(got, want) ** 2)) < (1e-5 if shell else 2e-6)


def test_fp32_direct_on_both_sides_of_the_kernels_rule(engine):
    """200,000 bodies run the row kernel, one more the tile kernel: each within
    the mode's 2e-6 rms of the FP64 sum."""
    b = scenarios.plummer(200_001, seed=5)
    big = engine.compute_forces(b.px, b.py, b.pz, b.mass, b.active, 1e-3, MODE_DIRECT)
    exact = engine.compute_forces(b.px, b.py, b.pz, b.mass, b.active, 1e-3, MODE_DIRECT_FP64)
    small = engine.compute_forces(b.px[:200_000], b.py[:200_000], b.pz[:200_000],
                                  b.mass[:200_000], b.active[:200_000], 1e-3, MODE_DIRECT)
    exact_small = engine.compute_forces(b.px[:200_000], b.py[:200_000], b.pz[:200_000],
                                        b.mass[:200_000], b.active[:200_000], 1e-3,
                                        MODE_DIRECT_FP64)
    assert np.sqrt(np.mean(rel_err(big, exact) ** 2)) < 2e-6
    assert np.sqrt(np.mean(rel_err(small, exact_small) ** 2)) < 2e-6
