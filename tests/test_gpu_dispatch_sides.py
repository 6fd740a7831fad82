"""Both sides of a dispatch rule compared bit for bit, where an input can be
made that runs the same sums on either; and the sizes beyond the other tests'."""
from __future__ import annotations

import numpy as np
import pytest

from nbody_b200 import (MODE_BARNES_HUT, MODE_DIRECT, MODE_DIRECT_FP64, B200PhysicsBackend,
                        B200SoAIntegrator, Engine, Ensemble, scenarios)
from nbody_b200 import _native as N
from test_gpu_shapes import test_keys_and_tree_at_dispatch_edges as check_keys_and_tree

pytestmark = pytest.mark.gpu

VECTORS = ("px", "py", "pz", "vx", "vy", "vz", "ax", "ay", "az")


def test_octree_numbering_with_scanned_block_sums(oracle):
    """More than 4096 numbering blocks of 1024 nodes each (4,194,304 nodes): the
    block sums are scanned by a kernel of their own."""
    n = 4_460_000  # 16 of 17 active
    with Engine(n) as e:
        check_keys_and_tree(e, oracle, n)


@pytest.mark.parametrize("span,bodies", [(0, 32), (256, 32), (256, 64)])
@pytest.mark.parametrize("eps", [1e-4, 0.0])
def test_walk_with_and_without_helping_warps(span, bodies, eps):
    """Two tree systems alone (few groups: idle warps help) and the same two in
    front of 480,000 other bodies (no helping): systems do not interact, so the
    two's forces are the same bits."""
    mine = [scenarios.plummer(k, seed=k) for k in (6000, 2500)]
    others = [scenarios.plummer(8192, seed=k) for k in range(58)]
    got = []
    for systems in (mine, mine + others):
        with Ensemble([b.n for b in systems], ds_max_n=2048) as e:
            e.set_param(N.PARAM_GROUP_SPAN, span)
            e.set_param(N.PARAM_GROUP_BODIES, bodies)
            e.set_state(systems)
            e.compute_forces(eps)
            s = e.get_state()
            got.append(np.array([s[k][:8500] for k in ("ax", "ay", "az")]))
    assert np.isfinite(got[0]).all() and (got[0] != 0).all()
    np.testing.assert_array_equal(got[0], got[1])


@pytest.mark.parametrize("n", [76_800, 87_040, 99_840])
def test_fp32_direct_kernels_give_the_same_bits(n):
    """Whole tiles of 2560 targets whose items leave their last wave too empty
    (0.963 to 0.966) run the row kernel.  With one body more, massless and in the
    last place of the Morton order (the corner of their box), a tile more fills
    it (0.991 to 0.995) and the tile kernel runs: over the same chunks of the same
    length at this capacity, adding exact zeros."""
    b = scenarios.plummer(n, seed=11)
    ext = {k: np.append(getattr(b, k), getattr(b, k).max()) for k in ("px", "py", "pz")}
    mass = np.append(b.mass, 0.0)
    act = np.ones(n + 1, np.uint8)
    with Engine(200_001) as e:
        for eps in (1e-3, 1e-6):
            few = e.compute_forces(b.px, b.py, b.pz, b.mass, b.active, eps, MODE_DIRECT)
            more = e.compute_forces(ext["px"], ext["py"], ext["pz"], mass, act, eps, MODE_DIRECT)
            for f, m in zip(few, more):
                np.testing.assert_array_equal(f, m[:n])


@pytest.mark.parametrize("order", ["simd", "pairwise", "shell"])
@pytest.mark.parametrize("n", [1, 2, 129, 295, 296, 297, 591, 592, 593, 1184, 1185])
def test_fp64_orders_in_every_block_shape(engine, oracle, n, order):
    """Forces and one-launch steps of the other summation orders and of the
    shell theorem, in blocks of 2, 4 and 8 targets: bit for bit the oracle's
    forces, and the Verlet step's operations one by one on them."""
    eps, dt = 1e-3, 1e-3
    if order == "shell" and n > 1:
        b = scenarios.collisional_disk(n, seed=n, radius_scale=3000.0)
    else:
        b = scenarios.plummer(n, seed=n)
    b.active[3::10] = 0
    shell = order == "shell"
    flag = MODE_DIRECT_FP64 | {"simd": N.FLAG_ORDER_SIMD, "pairwise": N.FLAG_ORDER_PAIRWISE,
                               "shell": N.FLAG_SHELL_THEOREM}[order]

    def forces(px, py, pz):
        return oracle.direct_forces_order(px, py, pz, b.mass, b.active, eps,
                                          {"simd": 1, "pairwise": 2, "shell": 0}[order],
                                          radius=b.radius, shell=shell)

    got = engine.compute_forces(b.px, b.py, b.pz, b.mass, b.active, eps, flag, radius=b.radius)
    for g, w in zip(got, forces(b.px, b.py, b.pz)):
        np.testing.assert_array_equal(g, w)
    live = b.active == 1
    for steps in (1, 2, 3):
        engine.set_state(b)
        engine.step(steps, dt, eps, flag)
        s, _ = engine.get_state()
        w = {k: np.array(getattr(b, k)) for k in VECTORS}
        for _ in range(steps):
            for x, v, a in (("px", "vx", "ax"), ("py", "vy", "ay"), ("pz", "vz", "az")):
                w[v][live] += 0.5 * dt * w[a][live]
                w[x][live] += dt * w[v][live]
            w["ax"], w["ay"], w["az"] = forces(w["px"], w["py"], w["pz"])
            for v, a in (("vx", "ax"), ("vy", "ay"), ("vz", "az")):
                w[v][live] += 0.5 * dt * w[a][live]
        for k in VECTORS:
            np.testing.assert_array_equal(getattr(s, k), w[k], err_msg=f"{k} {steps}")


@pytest.mark.parametrize("n", [1, 500, 20_000])
def test_integrator_writes_arrays_it_cannot_fill_in_place(n):
    """Strided, reversed, misaligned and single-precision arrays of the caller
    receive what contiguous ones do (rounded to their own type)."""
    plain = scenarios.plummer(n, seed=n)
    odd = plain.copy()
    odd.px = np.repeat(odd.px, 2)[::2]
    odd.vy = odd.vy[::-1].copy()[::-1]
    raw = np.zeros(8 * n + 1, np.uint8)
    odd.vz = raw[1:].view(np.float64)
    odd.vz[:] = plain.vz
    odd.az = odd.az.astype(np.float32)
    kept = {k: getattr(odd, k) for k in VECTORS}
    with Engine(n):
        back = B200PhysicsBackend(n, MODE_BARNES_HUT)
        for b in (plain, odd):
            B200SoAIntegrator().step(b, back, 1e-4, 1e-3, 3)
        back.engine.close()
    for k in VECTORS:
        assert getattr(odd, k) is kept[k]
        want = getattr(plain, k)
        np.testing.assert_array_equal(kept[k], want.astype(kept[k].dtype), err_msg=k)


def test_integrator_refuses_bodies_of_another_count_and_read_only_arrays():
    b = scenarios.plummer(300, seed=1)
    with Engine(300) as e:
        e.set_state(b)
        with pytest.raises(ValueError):
            e.get_vectors(scenarios.plummer(299, seed=1))
        b.vx.flags.writeable = False
        with pytest.raises(ValueError):
            e.get_vectors(b)
