"""1/sqrt in FP64: the routine of csrc/common.cuh over its whole range, and the
potential and the reference walk, which call the library's, at the ends of
theirs."""
from __future__ import annotations

import ctypes as C
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR
from nbody_b200 import MODE_BARNES_HUT_REF, scenarios
from nbody_b200 import _native as N

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "common.cuh"
__global__ void k(int n, const double* x, double* y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = nb::rsqrt_f64(x[i]);
}
extern "C" __attribute__((visibility("default"))) int run(int n, const double* x, double* y) {
    k<<<(n + 255) / 256, 256>>>(n, x, y);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def rsqrt_f64(tmp_path_factory):
    import torch

    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not (os.path.exists(nvcc) or shutil.which(nvcc)):
        pytest.skip("no nvcc on this machine")
    d = tmp_path_factory.mktemp("rsqrt")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--extended-lambda", "-shared", "-Xcompiler", "-fPIC", "-cudart", "shared",
                    "-I", str(PKG_DIR / "csrc"), "-I", str(PKG_DIR.parent / "include"),
                    "-o", str(d / "t.so"), str(d / "t.cu")], check=True)
    lib = C.CDLL(str(d / "t.so"))

    def f(x):
        dx = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        dy = torch.zeros_like(dx)
        torch.cuda.synchronize()
        assert lib.run(len(x), C.c_void_p(dx.data_ptr()), C.c_void_p(dy.data_ptr())) == 0
        return dy.cpu().numpy()

    return f


def test_every_exponent(rsqrt_f64):
    """The FP32 estimate y of x rounded to FP32 is off by at most 2^-22.5; the
    third-order step leaves 2.5 x that cubed, below 2^-66.  y y is exact (48
    bits), so the last fma's rounding, half a unit (2^-53 relative at most), is
    all but 2^-8 of the error inside the estimate's range.  The library's
    rsqrt, outside it, is good to one unit."""
    rng = np.random.default_rng(5)
    e = np.arange(-1074, 1024)
    m = np.concatenate([[1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52], 1.0 + rng.random(253)])
    with np.errstate(under="ignore"):
        x = np.ldexp(m[None, :], e[:, None]).ravel()
    x = np.concatenate([x, [1e-36, 1e36, np.nextafter(1e-36, 0), np.nextafter(1e36, 1e37)]])
    got = rsqrt_f64(x)
    want = 1 / np.sqrt(x.astype(np.longdouble))
    err = np.abs(got.astype(np.longdouble) - want) / want
    inside = (x >= 1e-36) & (x <= 1e36)
    assert err[inside].max() <= 2.0 ** -53 * (1 + 2.0 ** -8)
    assert err[~inside].max() <= 2.0 ** -52


def test_special_values(rsqrt_f64):
    got = rsqrt_f64(np.array([0.0, -0.0, np.inf, np.nan, -1.0, -np.inf, 5e-324]))
    assert got[0] == np.inf and got[1] == -np.inf and got[2] == 0.0
    assert np.isnan(got[3:6]).all()
    assert got[6] == pytest.approx(1 / math.sqrt(5e-324), rel=2.0 ** -51)


def _pair(d, mass):
    b = scenarios.plummer(2, seed=1)
    b.px, b.py, b.pz = np.array([0.0, d]), np.zeros(2), np.zeros(2)
    b.mass = np.array([mass, mass])
    return b


@pytest.mark.parametrize("exp", [-162, -160, -150, -100, -30, -18, 0, 18, 30, 100, 150, 153])
def test_potential_of_a_pair_at_any_distance(engine, exp):
    """-m^2 / d: d^2 (subnormal below 1e-154, with the bits it has left), its
    inverse root and two products, each within one unit."""
    d = 1.7 * 10.0 ** exp
    engine.set_state(_pair(d, 3.0))
    d2 = np.longdouble(d * d)
    assert engine.diagnostics(0.0)["pe"] == pytest.approx(float(-9 / np.sqrt(d2)), rel=2.0 ** -50)


def test_potential_of_a_coincident_pair(engine):
    engine.set_state(_pair(0.0, 1.0))
    assert engine.diagnostics(0.0)["pe"] == -np.inf
    assert engine.diagnostics(0.25)["pe"] == pytest.approx(-4.0, rel=2.0 ** -51)


@pytest.mark.parametrize("exp", [-90, -60, -18, 0, 18, 60, 90])
def test_reference_walk_of_a_pair_at_any_distance(engine, exp):
    """m / d^2 towards the other body: as above, with two products more."""
    d = 1.7 * 10.0 ** exp
    b = _pair(d, 3.0)
    ax, ay, az = engine.compute_forces(b.px, b.py, b.pz, b.mass, b.active, 0.0,
                                       MODE_BARNES_HUT_REF)
    want = 3.0 / d / d
    np.testing.assert_allclose(ax, [want, -want], rtol=2.0 ** -49)
    assert not ay.any() and not az.any()


@pytest.mark.parametrize("radius", [0.0, 1.0])
def test_reference_walk_shell_leaf_beyond_the_cube_roots_range(engine, radius):
    """Heavy bodies so far apart that 1/d^3 is subnormal but m/d^3 is not: the
    leaf's coefficient is built one factor at a time, each within one unit."""
    b = _pair(1.7e105, 3e60)
    b.radius = np.full(2, radius)
    ax, _, _ = engine.compute_forces(b.px, b.py, b.pz, b.mass, b.active, 0.0,
                                     MODE_BARNES_HUT_REF | N.FLAG_SHELL_THEOREM, radius=b.radius)
    want = 3e60 / 1.7e105 / 1.7e105
    np.testing.assert_allclose(ax, [want, -want], rtol=2.0 ** -49)
