"""The transfers between the caller's arrays and the device (csrc/hostio.cu)
on the CPU, over a runtime of plain memory that counts pins and copies."""
from __future__ import annotations

import ctypes as C
import multiprocessing
import os
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from conftest import PKG_DIR

MB = 1 << 20
CUDA_INCLUDE = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    if not shutil.which("g++") or not (CUDA_INCLUDE / "cuda_runtime.h").exists():
        pytest.skip("no g++ or no CUDA headers")
    so = tmp_path_factory.mktemp("hostio") / "hostio_fake.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-shared", "-fPIC", "-pthread",
                    "-Wl,-Bsymbolic",  # its own runtime, whatever else is loaded
                    "-I", str(PKG_DIR / "csrc"), "-I", str(CUDA_INCLUDE), "-x", "c++", "-o", str(so),
                    str(Path(__file__).parent / "hostio_fake.cpp")], check=True)
    return so


class Host:
    """One loaded copy of the library, with counters of its own."""

    def __init__(self, so, tmp_path):
        own = tmp_path / "own.so"  # a path of its own: dlopen shares by path
        shutil.copy(so, own)
        self.lib = lib = C.CDLL(str(own))
        lib.t_open.restype, lib.t_open.argtypes = C.c_void_p, [C.c_int, C.c_size_t]
        lib.t_close.argtypes = [C.c_void_p]
        for f in (lib.t_up, lib.t_down):
            f.argtypes = [C.c_void_p, C.c_int, C.POINTER(C.c_void_p), C.POINTER(C.c_void_p),
                          C.c_size_t]

    def open(self, row_bytes=8 * MB, rows=14):
        h = self.lib.t_open(rows, row_bytes)
        assert h
        return h

    def counts(self):
        out = (C.c_size_t * 5)()
        self.lib.t_counts(out)
        return dict(zip(("pinned", "pinned_ever", "pins", "copies", "pinned_copies"), out))

    def move(self, f, h, dst, src):
        def ptrs(a):
            return (C.c_void_p * len(a))(*(x.ctypes.data for x in a))

        before = self.counts()
        assert f(h, len(dst), ptrs(dst), ptrs(src), dst[0].nbytes) == 0
        after = self.counts()
        for d, s in zip(dst, src):
            np.testing.assert_array_equal(d, s)
        return {k: after[k] - before[k] for k in after}

    def up(self, h, total, rows=12, seed=0):
        """`rows` arrays of `total` bytes in all: what the call counted."""
        b = max(8, total // rows // 8 * 8)
        src = [np.random.default_rng(seed + k).integers(0, 255, b).astype(np.uint8)
               for k in range(rows)]
        return self.move(self.lib.t_up, h, [np.zeros_like(a) for a in src], src)

    def down(self, h, total, rows=12, seed=0):
        b = max(8, total // rows // 8 * 8)
        src = [np.random.default_rng(seed + k).integers(0, 255, b).astype(np.uint8)
               for k in range(rows)]
        return self.move(self.lib.t_down, h, [np.zeros_like(a) for a in src], src)

    def warm(self, h):
        """Moves enough for the pool to be there with all its slots."""
        for _ in range(20):
            self.down(h, 4 * MB)


@pytest.fixture
def host(built, tmp_path):
    return Host(built, tmp_path)


POOL = pytest.mark.skipif(len(os.sched_getaffinity(0)) < 6, reason="too few CPUs for the pool")


@POOL
def test_uploads_below_the_pools_line_are_plain_copies(host):
    """Up to 28 MB the plain copy of an upload is as fast as the pool or
    faster (12 MB 0.56 against 1.24 ms); downloads go by the pool from 2 MB."""
    h = host.open()
    host.warm(h)
    for mb in (1, 4, 12, 27):
        c = host.up(h, mb * MB)
        assert c["copies"] == 12 and c["pinned_copies"] == 0, mb
    c = host.up(h, 30 * MB)
    assert c["copies"] >= 12 and c["pinned_copies"] == c["copies"]
    c = host.down(h, 3 * MB)
    assert c["copies"] >= 12 and c["pinned_copies"] == c["copies"]
    host.lib.t_close(h)
    assert host.counts()["pinned"] == 0


def test_a_handle_without_pinned_memory_still_transfers(host):
    host.lib.t_refuse_pins(1)
    h = host.open()
    for total in (96, 60_000, 3 * MB, 40 * MB):
        for f in (host.up, host.down):
            assert f(h, total)["pinned_copies"] == 0
    host.lib.t_refuse_pins(0)
    other = host.open()
    assert host.up(other, 60_000)["pinned_copies"] > 0
    host.lib.t_close(h)
    host.lib.t_close(other)
    assert host.counts()["pinned"] == 0


@pytest.mark.parametrize("n", [1, 64, 1000, 4681, 4700, 1 << 20])
def test_a_handle_pins_what_its_largest_transfer_needs(host, n):
    """Two halves (up, down) of 14 arrays of n doubles, in whole pages and at
    most 512 KB each, and 4 KB; the largest transfer is one that fits."""
    h = host.open(8 * n)
    rows = -(-8 * n // 256) * 256 * 14
    half = min(512 << 10, -(-rows // 4096) * 4096)
    assert host.counts()["pinned"] == 2 * half + 4096
    for f in (host.up, host.down):
        c = f(h, 14 * 8 * n, rows=14)
        if rows <= half:
            assert c["pinned_copies"] == c["copies"] == 14
    host.lib.t_close(h)
    assert host.counts()["pinned"] == 0


def test_a_handle_that_wants_no_pinned_memory_pins_none(host):
    h = host.open(8 * 1000, rows=0)
    assert host.counts()["pins"] == 0
    assert host.up(h, 9000)["pinned_copies"] == host.down(h, 9000)["pinned_copies"] == 0
    host.lib.t_close(h)


def test_a_closed_handles_pinned_memory_goes_to_the_next_that_fits(host):
    keep = host.open(8 * 64)
    small, large = host.open(8 * 500), host.open(8 * 100_000)
    pins = host.counts()["pins"]
    host.lib.t_close(small)
    host.lib.t_close(large)
    again = host.open(8 * 100_000)  # the small one's is too small for it
    assert host.counts()["pins"] == pins
    host.up(again, 400_000)
    host.down(again, 400_000)
    tiny = host.open(8 * 400)
    assert host.counts()["pins"] == pins
    many = [host.open(8 * 300) for _ in range(12)]
    for h in (again, tiny, *many):
        host.lib.t_close(h)
    host.lib.t_close(keep)
    assert host.counts()["pinned"] == 0


def _on_few_cpus(so, path, cpus):
    os.sched_setaffinity(0, sorted(os.sched_getaffinity(0))[:cpus])
    host = Host(so, path)
    h = host.open(8 * 64)
    own = host.counts()["pinned"]
    host.warm(h)
    host.up(h, 60 * MB)
    assert host.counts()["pinned"] == own
    host.lib.t_close(h)


@pytest.mark.parametrize("cpus", [1, 5])
def test_too_few_cpus_for_the_pool_pin_nothing_for_it(built, tmp_path, cpus):
    """A pool of fewer than two threads is never used, so its slots are not pinned."""
    p = multiprocessing.get_context("spawn").Process(target=_on_few_cpus,
                                                     args=(built, tmp_path, cpus))
    p.start()
    p.join(120)
    assert p.exitcode == 0


@POOL
@pytest.mark.parametrize("mb", [3, 40])
def test_the_pools_slots_come_a_few_at_a_time(host, mb):
    """No call pins more than the first 4 MB, and the pool works from then on,
    while it grows to 16 MB."""
    h = host.open(8 * 64)
    own = host.counts()["pinned"]
    pinned = []
    for _ in range(24):
        c = host.down(h, mb * MB)
        pinned.append(c["pinned"])
        assert (c["pinned_copies"] > 0) == (sum(pinned) > 0)
    first = pinned.index(4 * MB)
    assert first * mb < 32 <= (first + 1) * mb
    assert pinned[first + 1:first + 8] == [2 * MB] * 6 + [0]
    host.up(h, 60 * MB)
    assert host.counts()["pinned"] == own + 16 * MB
    host.lib.t_close(h)
    assert host.counts()["pinned"] == 0


@POOL
def test_a_pool_that_gets_no_slots_leaves_the_plain_copy(host):
    h = host.open(8 * 64)
    host.lib.t_refuse_pins(1)
    host.warm(h)
    assert host.down(h, 8 * MB)["pinned_copies"] == 0
    host.lib.t_refuse_pins(0)
    assert host.down(h, 8 * MB)["pinned_copies"] == 0
    host.lib.t_close(h)


def test_pinned_memory_is_not_inherited_by_child_processes(host):
    """A fork must not turn the pages that the device knows into copies: the
    mapping carries the kernel's do-not-copy flag."""
    h = host.open(8 * 1000)
    out = (C.c_size_t * 2)()
    host.lib.t_some_pinned(out)
    start, size = out
    flags = None
    for line in Path("/proc/self/smaps").read_text().splitlines():
        head = line.split()[0]
        if "-" in head and not head.endswith(":"):
            lo, hi = (int(x, 16) for x in head.split("-"))
            inside = lo <= start and start + size <= hi
        elif head == "VmFlags:" and inside:
            flags = line.split()[1:]
    assert flags is not None and "dc" in flags
    host.lib.t_close(h)
