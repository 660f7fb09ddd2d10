"""Deposits a rounding away from a face of the voxel that hit a sphere one past the lattice: its key is
that of a sphere in the next row or layer, a voxel away, and the reference sums the two as one. Such
deposits stand at the front and the end of a track, in every layer, so windows of the track or of its
layers would part some. Hits, spheres and counts bit-exact against the CPU oracle, y*f(y) within 1e-12."""
import numpy as np
import pytest

import pyoracle as po
import supertrack_b200 as st
from helpers import assert_hist_equal, assert_stats_equal

pytestmark = pytest.mark.gpu

HL, D, N_OS, SEED = 1000.0, 10.0, 4, 9
GSO = -HL + D / 2


def _before(value, shift):
    """A coordinate that the shift takes exactly to `value`."""
    c = value - shift
    for k in range(-4, 5):
        t = c
        for _ in range(abs(k)):
            t = np.nextafter(t, np.inf * np.sign(k))
        if t + shift == value:
            return t
    raise ValueError("no such coordinate")


def _track(axis, sx, sy):
    """Deposits along z, and in front and behind, for every layer, the two of a pair that wraps on an
    axis's upper face."""
    rs = np.random.default_rng(3)
    n, pairs = 24_000, range(10, 190)
    p = np.stack([*rs.normal(scale=10.0, size=(2, n)), np.sort(rs.uniform(-HL, HL, n))])
    for c, kz in enumerate(pairs):
        a = GSO + D * np.array([100.0, 100.0, kz])
        b = a.copy()
        a[axis] = np.nextafter(HL, 0)
        # the sphere whose key it takes: the first of the next row or layer
        b[axis] = GSO
        b[axis + 1] += D
        for at, pair in ((c, a), (-1 - c, b + 0.25)):
            p[:, at] = [_before(pair[0], sx), _before(pair[1], sy), pair[2]]
    e = np.clip(np.exp(np.log(20) + 0.8 * rs.normal(size=n)), 10, 1000)
    return [np.ascontiguousarray(v) for v in (*p, e)]


@pytest.mark.parametrize("bins", [200, 3000])       # the 8192- and the 4096-slot table
@pytest.mark.parametrize("sort", [0, 1])            # boundary flags, layers
@pytest.mark.parametrize("shift_track", [False, True])
@pytest.mark.parametrize("axis", [0, 1])
def test_wrapped_keys(ctx, axis, shift_track, sort, bins):
    sxsy = st.oversample_shifts(HL, D, shift_track, SEED, 1, N_OS)
    t = _track(axis, *np.asarray(sxsy).reshape(-1, 2)[1])
    spec = ("log", bins, 0.01, 1e5)
    oc, oy = np.zeros(bins, dtype=np.int64), np.zeros(bins)
    _, _, os_, _ = po.run_job(*t, half_length=HL, sphere_diameter=D, sxsy=sxsy,
                              edges_arr=po.edges(*spec), zshift="none", counts=oc, yfy=oy)
    old = ctx.get_param("sort_deposits")
    ctx.set_param("sort_deposits", sort)
    try:
        ctx.clear()
        hid = ctx.histogram(*spec)
        jid = ctx.submit(*t, half_length=HL, sphere_diameter=D, n_oversamples=N_OS, hist=hid,
                         seed=SEED, track_id=1, zshift="none", shift_track=shift_track)
        ctx.run()
        gc, gy = ctx.read_histogram(hid)
        gs = ctx.stats(jid)
    finally:
        ctx.set_param("sort_deposits", old)
    assert_stats_equal([gs], [os_])
    assert_hist_equal([gc], [gy], [oc], [oy])
