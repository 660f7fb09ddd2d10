"""The device code that cuts a batch into work (planning.cuh), compiled for the host and run with its
warps in other orders than a GPU usually takes: one warp at a time from barrier to barrier."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from supertrack_b200 import _capi

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    out = str(tmp_path_factory.mktemp("emulated") / "libplanning.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-fPIC", "-shared", "-ffp-contract=off",
                    "-isystem", include, os.path.join(HERE, "planning_on_cpu.cc"), "-o", out],
                   check=True)
    return C.CDLL(out)


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


ORDERS = {"first warp first": np.arange(32), "last warp first": np.arange(32)[::-1],
          "second warp first": np.roll(np.arange(32), -1),
          "odd warps first": np.concatenate([np.arange(1, 32, 2), np.arange(0, 32, 2)])}


def _order(name):
    o = ORDERS[name]
    return np.concatenate([o, o[o < 4]]).astype(np.int32)


# batches whose items fall into one bucket, into both halves of the buckets, and the sizes at which
# the items are written by the planning CTA or by a second launch
BATCHES = {
    "one short track": [(4000, 10)],
    "64 equal tracks": [(4000, 10)] * 64,
    "65 equal tracks": [(4000, 10)] * 65,
    "uneven": [(int(4 ** (1 + k % 9)) + k, 1 + 7 * (k % 5)) for k in range(60)],
    "empty ones between": [(0, 10), (3000, 0), (128, 1), (0, 0), (70_000, 3)],
    "one item of 2^33 and many small": [(1 << 33, 1)] + [(500, 4)] * 20,
}


@pytest.mark.parametrize("order", sorted(ORDERS))
@pytest.mark.parametrize("batch", sorted(BATCHES))
def test_plan_covers_every_oversample_once(lib, batch, order):
    jobs = BATCHES[batch]
    kept = np.array([k for k, _ in jobs], dtype=np.int64)
    n_os = np.array([o for _, o in jobs], dtype=np.int32)
    cap = int(n_os.sum()) * 32 + 8
    items = np.zeros((cap, 6), dtype=np.int32)
    n = lib.plan_batch(len(jobs), _ptr(kept), _ptr(n_os), 148, C.c_int64(1 << 18), 0,
                       C.c_int64(cap), _ptr(_order(order)), _ptr(items))
    done = [np.zeros(o, dtype=int) for o in n_os]
    cost = []
    for job, first, count, unit, _, _ in items[:n]:
        assert 0 <= job < len(jobs) and unit < 0 and count > 0
        done[job][first:first + count] += 1
        cost.append(int(kept[job]) * int(count))
    for k, d in zip(kept, done):
        assert np.all(d == (1 if k else 0))
    # longest first, to within a factor of two and the padding to whole tiles
    assert all(a * 4 + 1024 >= b for a, b in zip(cost, cost[1:]))
    assert np.all(items[n:] == -1)


@pytest.mark.parametrize("order", sorted(ORDERS))
@pytest.mark.parametrize("per_window", [1, 33, 700, 1024])
def test_threads_agree_when_a_table_is_emptied(lib, per_window, order):
    """Also at a window that ends with the count at, or one above, the limit."""
    for limit in (2 * per_window, 2 * per_window - 1, 3 * per_window - 1):
        assert lib.empty_windows(40, per_window, limit, _ptr(_order(order))) == 0


@pytest.mark.parametrize("ratio_bits", [0, 1, 11, 31, 41, 42, 43, 54, 55, 56, 57, 73, 74, 100])
@pytest.mark.parametrize("lower", [1e-30, 0.01, 3.0])
@pytest.mark.parametrize("work", [1, 2048, 1 << 18, (1 << 18) + 1, 4_000_000, 1 << 33])
def test_kept_sums_stay_below_128_bits(lib, ratio_bits, lower, work):
    """The y*f(y) sum of a bin in shared memory, at the most spheres and the largest y that are
    added to it between two flushes, comes back from its 128-bit form as it is."""
    lower = float(np.float32(lower))
    edges = np.array([lower, lower * 1.7 * 2.0 ** ratio_bits, lower * 4.0 * 2.0 ** ratio_bits])
    bits = lib.keep_bits(_ptr(edges), 2)
    span = lib.sum_span(bits, C.c_int64(work))
    assert 18 <= bits <= 31 and span >= 12     # (an offset below 12 is not compared with the span)
    if ratio_bits <= 40:
        assert bits == 31
    spheres = max(work, 1 << bits)
    for b in range(2):
        y = np.nextafter(edges[b + 1], 0.0)
        up = int(np.frexp(y)[1] - np.frexp(edges[b])[1])
        if up > span:
            assert up > 55 or work > 1 << 18
            y, up = float(np.ldexp(2.0 - 2.0 ** -52, int(np.frexp(edges[b])[1]) - 1 + span)), span
        e0 = int(np.frexp(edges[b])[1]) - 53    # exponent of the lower edge's last place
        lo, hi = C.c_uint64(), C.c_uint64()
        _capi.lib().st_to_fixed(float(y), e0, C.byref(lo), C.byref(hi))
        total = ((hi.value << 64) | lo.value) * spheres
        assert total < 1 << 127
        back = _capi.lib().st_from_fixed(total & (2 ** 64 - 1), total >> 64, e0)
        assert back == float(y) * spheres
