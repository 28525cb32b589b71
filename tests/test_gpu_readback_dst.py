"""Where particle arrays are read to: fresh, used, half-used and misaligned
pageable memory, page-locked memory, and two threads at once."""
import ctypes as C
import mmap
import threading
import time

import numpy as np
import pytest

from ziran2019_b200 import abi, mpm

pytestmark = pytest.mark.gpu

DX = 1.0 / 256
KEYS = "XVCF"


def make(n, seed=0):
    rng = np.random.default_rng(seed)
    s = mpm.MpmSimulation(DX, precision="mixed", grid_log2=8)
    s.addParticles(0.3 + 0.4 * rng.random((n, 3)), None, 1.0, 1.0)
    a = {"X": 0.3 + 0.4 * rng.random((n, 3)), "V": rng.standard_normal((n, 3)), "C": rng.standard_normal((n, 3, 3)),
         "F": rng.standard_normal((n, 3, 3))}
    s.binParticles()
    s.setParticles(**a)
    s.binParticles()
    return s, a


def read(s, ptrs):
    assert s.lib.get_particles(s.ctx, *[C.cast(p, abi.c_double_p) if p else None for p in ptrs]) == abi.OK


def mapped(nbytes, kind):
    """Memory from mmap (no page of it touched yet): as it is, all touched, every third page touched."""
    m = mmap.mmap(-1, nbytes + 4096)
    b = np.frombuffer(m, dtype=np.uint8)
    if kind == "used":
        b[:] = 7
    if kind == "half":
        b[::3 * 4096] = 7
    return b


# C and F (72 n bytes) around 8 MB, where fresh pages are touched first; X and V (24 n) too
@pytest.mark.parametrize("n", [3, 116508, 116509, 349525, 349526, 500003])
@pytest.mark.parametrize("kind,shift", [("fresh", 0), ("fresh", 8), ("used", 0), ("half", 8)])
def test_pageable(cuda_lib, n, kind, shift):
    s, a = make(n, n)
    size = {k: a[k].nbytes for k in KEYS}
    dst = {k: mapped(size[k] + shift + 64, kind) for k in KEYS}
    tail = {k: dst[k][shift + size[k]:].copy() for k in KEYS}
    read(s, [dst[k].ctypes.data + shift for k in KEYS])
    for k in KEYS:
        np.testing.assert_array_equal(dst[k][shift:shift + size[k]].view(np.float64), a[k].ravel())
        np.testing.assert_array_equal(dst[k][shift + size[k]:], tail[k])  # nothing past the array
        assert not dst[k][:shift].any() or kind != "fresh"


def test_some_arrays_only(cuda_lib):
    s, a = make(400000, 1)
    dst = {k: mapped(a[k].nbytes, "fresh") for k in "VF"}
    read(s, [dst[k].ctypes.data if k in dst else None for k in KEYS])
    for k in dst:
        np.testing.assert_array_equal(dst[k][:a[k].nbytes].view(np.float64), a[k].ravel())


def test_page_locked_runs_at_the_link_rate(cuda_lib):
    """One direct transfer per array: at most twice what the same bytes take as plain transfers into the same memory
    (through staging blocks they took 3.2 times as long)."""
    import torch
    n = 500000
    s, a = make(n, 2)
    pin = {k: torch.empty(a[k].shape, dtype=torch.float64, pin_memory=True) for k in KEYS}
    dev = {k: torch.empty(a[k].shape, dtype=torch.float64, device="cuda") for k in KEYS}

    def best(f):
        t = []
        for _ in range(9):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            f()
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        return min(t)

    plain = best(lambda: [pin[k].copy_(dev[k], non_blocking=True) for k in KEYS])
    ours = best(lambda: read(s, [pin[k].data_ptr() for k in KEYS]))
    for k in KEYS:
        np.testing.assert_array_equal(pin[k].numpy(), a[k])
    assert ours <= 2 * plain, (ours, plain)


def test_two_threads(cuda_lib):
    """Two contexts read at the same time, each into fresh memory, several times."""
    pairs = [make(400000 + 17 * i, 5 + i) for i in range(2)]
    bad = []

    def work(s, a):
        for _ in range(4):
            b = s.getParticles()
            bad.extend(k for k in KEYS if not np.array_equal(a[k], b[k]))

    threads = [threading.Thread(target=work, args=p) for p in pairs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
