"""The device code that cuts a batch into work (planning.cuh), compiled for the host and run with its
warps in other orders than a GPU usually takes: one warp at a time from barrier to barrier."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from supertrack_b200 import _capi
from test_integer_geometry_property import _deposits, _fp64, _geometry

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
    items = np.zeros((cap, 4), dtype=np.int32)
    n = lib.plan_batch(len(jobs), _ptr(kept), _ptr(n_os), _ptr(np.zeros_like(n_os)), 148, C.c_int64(1 << 18), 0,
                       C.c_int64(cap), _ptr(_order(order)), _ptr(items))
    done = [np.zeros(o, dtype=int) for o in n_os]
    cost = []
    for job, first, count, unit in items[:n]:
        assert 0 <= job < len(jobs) and unit < 0 and count > 0
        done[job][first:first + count] += 1
        cost.append(int(kept[job]) * int(count))
    for k, d in zip(kept, done):
        assert np.all(d == (1 if k else 0))
    # longest first, to within a factor of two and the padding to whole tiles
    assert all(a * 4 + 1024 >= b for a, b in zip(cost, cost[1:]))
    assert np.all(items[n:] == -1)


@pytest.mark.parametrize("grid", [1, 4, 148])
@pytest.mark.parametrize("kept,n_os,n_win", [(20_000, 4, 3), (20_000, 400, 1), (300_007, 10, 74),
                                            (4_000_000, 4, 1), (4_000_000, 3, 977),
                                            (4_000_000, 50, 33), (300_000, 7, 2)])
def test_plan_covers_every_window_once(lib, kept, n_os, n_win, grid):
    """A layered job's items are whole oversamples, or parts of one that cover all its windows."""
    cap = n_os * 32
    items = np.zeros((cap, 4), dtype=np.int32)
    n = lib.plan_batch(1, _ptr(np.array([kept])), _ptr(np.array([n_os], dtype=np.int32)),
                       _ptr(np.array([n_win], dtype=np.int32)), grid, C.c_int64(1 << 18), 8,
                       C.c_int64(cap), _ptr(_order("first warp first")), _ptr(items))
    done = np.zeros((n_os, n_win), dtype=int)
    for job, first, count, unit in items[:n]:
        assert job == 0 and unit < 0
        if count > 0:
            assert unit == -1
            done[first:first + count] += 1
        else:
            done[first, -count * (-1 - unit):-count * -unit] += 1
    assert np.all(done == 1)


NONE, FLAGS, LAYERS = range(3)
# z bins, deposits per sphere diameter, deposit*oversamples per CTA, mode
TRACKS = {
    "along z": ([300] * 1000, 3000.0, 20_000, LAYERS),
    "few deposits": ([16_384], 3000.0, 20_000, NONE),
    "dense, in one bin, 4 oversamples": ([900_000] + [1000] * 100, 3000.0, 27_000, FLAGS),
    "the same with shared units off": ([900_000] + [1000] * 100, 3000.0, 27_000, LAYERS),
    "the same, 148 oversamples": ([900_000] + [1000] * 100, 3000.0, 1_000_000, LAYERS),
    "dense, in two bins, 10 oversamples": ([135_000] * 2 + [300] * 100, 1800.0, 20_000, FLAGS),
    "dense, in two bins, large": ([900_000] * 2 + [2000] * 100, 4000.0, 54_000, LAYERS),
    "dense, in eight bins": ([40_000] * 8, 1800.0, 8_000, LAYERS),
    "dense, in one bin, too small for units": ([120_000], 1800.0, 3_000, LAYERS),
    "sparse, a third in large bins": ([400] * 300 + [20_000] * 3, 500.0, 5_000, FLAGS),
    "sparse, a fifth in large bins": ([400] * 300 + [30_000], 500.0, 5_000, LAYERS),
}


@pytest.mark.parametrize("order", sorted(ORDERS))
@pytest.mark.parametrize("track", sorted(TRACKS))
def test_window_mode(lib, track, order):
    """Layers, unless they would leave most CTAs without work or empty bins into the log."""
    sizes, per_d, share, mode = TRACKS[track]
    bins = np.array(sizes, dtype=np.uint32)
    unit_min = (1 << 62) if "units off" in track else 4 * 32_768
    assert lib.window_mode(len(bins), _ptr(bins), C.c_double(per_d), C.c_int64(share),
                           C.c_int64(unit_min), _ptr(_order(order))) == mode
    if sum(sizes) > 16_384:
        assert np.array_equal(bins, np.concatenate([[0], np.cumsum(sizes)[:-1]]))


def test_footprint_charges_what_a_job_allocates(lib):
    """st_server_job_footprint against the arrays of a context that grow with a job; and no more
    than 48 bytes of records per deposit and 8 of a qualifying job's shifted z came to, so that what
    a budget admitted is still admitted."""
    size = np.zeros(7, dtype=np.int64)
    lib.sizes(_ptr(size))
    job, aux, plan, hist, item, slot, record = [int(v) for v in size]
    lib.window_cap.restype = C.c_int64
    for n, d, n_os, nbins in [(1, 10.0, 1, 1), (1000, 10.0, 65_536, 4096), (8192, 2.0, 100, 200),
                              (8193, 2.0, 100, 200), (8193, 1.0, 4, 200), (20_001, 1.3, 4, 3000),
                              (1_000_000, 2.0, 100, 500), (4_000_000, 10.0, 50, 3000),
                              (100_000, 1000.0, 50, 200), (200_000, 30.0, 4, 7)]:
        hl = 2500.0
        lattice = int(2 * hl / d)
        pad, blocks = -(-n // 128) * 128, -(-n // 1024)
        want = (32 * n + record * pad + job + aux + plan + hist + blocks * (8 + 4 + 4) + 8
                + n_os * (32 * item + 3 * 4) + 16 * nbins + 8 * (nbins + 1))
        if n > 8192 and n_os >= 4 and 128 <= lattice < 1 << 19:
            cells = 1 << (2 * n - 1).bit_length()
            bins = lattice
            while bins > 4096:
                bins = (bins + 1) // 2
            # cell hash, z bins, window list (of windows on the smaller table)
            want += slot * cells + 4 * bins + 8 * lib.window_cap(C.c_int64(n), C.c_int64(4096))
        view, desc, got = _capi.st_track_view(), _capi.st_job_desc(), C.c_int64(0)
        view.n, view.on_device = n, 1
        desc.half_length, desc.sphere_diameter, desc.n_oversamples = hl, d, n_os
        assert _capi.lib().st_server_job_footprint(C.byref(view), C.byref(desc), nbins,
                                                   C.byref(got)) == 0
        assert got.value >= want
        pad256 = -(-n // 256) * 256
        flagged = n > 8192 and n_os >= 4 and 128 <= lattice < 1 << 19
        most = (32 * n + 48 * pad256 + 24 * nbins + 8 + 512 + 524 * n_os
                + ((16 * (1 << (2 * n - 1).bit_length()) + 8 * pad256) if flagged else 0))
        assert got.value <= most


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


@pytest.mark.parametrize("kind,nbins,lower,upper", [
    ("lin", 3000, 0.01, 300.0), ("log", 500, 0.1, 1e4), ("lin", 1, 1e-13, 1e4), ("lin", 3, 1e-20, 9.0),
    ("log", 4, 1e-30, 1e30), ("log", 4096, 1e-30, 1e30), ("lin", 10, 0.0, 1.0), ("lin", 7, -3.0, 4.0),
    ("lin", 2, -1.0, 1.0), ("lin", 1, -2.0, -1.0)])
def test_keep_bits_of_histograms(lib, kind, nbins, lower, upper):
    """The widest bin with a positive normal lower edge decides how long a copy is kept."""
    edges = np.zeros(nbins + 1)
    _capi.check(_capi.lib().st_hist_edges({"lin": _capi.ST_HIST_LIN, "log": _capi.ST_HIST_LOG}[kind], nbins, lower, upper,
                                          _ptr(edges)), "st_hist_edges")
    e = np.frexp(edges)[1]
    wide = [int(b - a) for a, b, lo in zip(e, e[1:], edges) if lo >= 2.0 ** -1022]
    assert lib.keep_bits(_ptr(edges), nbins) == min(31, max(18, 73 - max(wide, default=0)))


@pytest.mark.parametrize("win_tiles", [32, 64])
@pytest.mark.parametrize("m", [1, 3, 4, 5, 8, 100])
def test_window_list(lib, m, win_tiles):
    """cut_windows: windows that follow one another, end at the end of a bin or, inside one, at a
    whole tile (the next one is then marked), span no more tiles than they may, and fit the arena."""
    rng = np.random.default_rng(win_tiles * 100 + m)
    tiles = (1 if m < 2 else 2 if m < 4 else min(m, 8)) * win_tiles
    lists = [np.full(4096, s) for s in (1, 5, 127, 128, 129, 1000)]
    for a in (1, 21, 22, 31, 32, 33, win_tiles):
        for big in (12, 34, win_tiles + 1, 8 * win_tiles + 1):
            lists.append(np.tile([a * 128, big * 128], 40))
            lists.append(np.tile([a * 128 + 1, 0, big * 128 - 1, 3], 40))
    for _ in range(20):
        lists.append(rng.integers(0, 2 ** rng.integers(1, 18), size=rng.integers(1, 600)) + 1)
        lists.append((rng.pareto(0.8, size=300) * 200).astype(np.int64) % 300_000 + 1)
    lib.window_cap.restype = C.c_int64
    for sizes in lists:
        ends = np.cumsum(sizes).astype(np.uint32)
        kept = int(ends[-1])
        cap = lib.window_cap(C.c_int64(kept), C.c_int64(win_tiles * 128))
        wins = np.zeros(2 * cap + 64, dtype=np.uint64)
        n = lib.cut(len(ends), _ptr(ends), C.c_int64(max(kept // m, 1)), win_tiles, _ptr(wins))
        assert n + 1 <= cap
        first = (wins[:n + 1] & np.uint64(2 ** 63 - 1)).astype(np.int64)
        inside = wins[:n + 1] >= np.uint64(2 ** 63)
        assert first[0] == 0 and first[n] == kept and np.all(np.diff(first) > 0)
        assert not inside[0] and not inside[n]
        assert np.all(-(-first[1:] // 128) - first[:-1] // 128 <= tiles)
        at_end = np.isin(first[1:], ends)
        # (a cut inside a bin falls on a whole tile, which may happen to be a bin's end as well)
        assert np.all(at_end | inside[1:]) and np.all(first[1:][inside[1:]] % 128 == 0)


@pytest.mark.parametrize("hl,d", [(2500.0, 2.0), (2500.0, 1000.0), (5000.0, 10.0), (1.0, 2.0),
                                  (3.0, 1000.0), (1e6, 1.0), (0.37, 1e-3), (5e12, 7e6)])
def test_integer_geometry_with_the_kernel_constants(lib, hl, d):
    """What set_integer_geometry lets the 32-bit integers and float sums decide, FP64 decides too."""
    rs = np.random.default_rng(int(hl * 7 + d * 13) % 2 ** 32)
    n, h, length, gso = _geometry(hl, d)
    for u in (1.0, 2.0 ** -24, 0.5, *rs.random(3)):
        sx, sy = u * length - h, rs.random() * length - h
        x, y, dz = _deposits(rs, n, h, d, gso, sx, sy, 60_000)
        out = [np.zeros(len(x), dtype=np.int32) for _ in range(3)]
        f = C.c_double
        lib.integer_geometry(len(x), C.c_int64(n), f(d), f(gso), f(sx), f(sy), _ptr(x), _ptr(y),
                             _ptr(dz), *[_ptr(o) for o in out])
        inb, hit, kx, ky = _fp64(x, y, dz, sx, sy, h, d, gso)
        sure = out[0] & 4 == 0
        assert np.array_equal((out[0] & 1 != 0)[sure], inb[sure])
        found = sure & (out[0] & 2 != 0)
        assert np.array_equal(found[sure], hit[sure])
        assert np.array_equal(out[1][found], kx[found]) and np.array_equal(out[2][found], ky[found])
        assert found.sum() > len(x) // 100
