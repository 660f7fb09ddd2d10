"""Dense tracks (over 1,024 deposits per sphere diameter) across z and nearly so, with few oversamples:
nearly all deposits in two z bins or in one (boundary flags and shared units, or layers where one CTA
runs the batch), in several bins larger than a window, in large and small ones (layers); on one CTA, a
few and all; few helpers; both tables and precisions. Hits, spheres, binned spheres and counts
bit-exact against the CPU oracle, y*f(y) within 1e-12."""
import numpy as np
import pytest

import pyoracle as po
import supertrack_b200 as st
from helpers import assert_hist_equal, assert_stats_equal

pytestmark = pytest.mark.gpu

HL, N_OS = 300.0, 4


def _track(n, tilt, core, slab, seed):
    """n deposits along a line that makes an angle `tilt` with the x axis, the last `slab` of them
    spread over one layer instead."""
    rs = np.random.default_rng(seed)
    t = np.sort(rs.uniform(-HL, HL, n))
    r = np.where(rs.random(n) < 0.7, core * np.abs(rs.normal(size=n)), core * 30 ** rs.random(n))
    a = rs.uniform(0, 2 * np.pi, n)
    p, q = r * np.cos(a), r * np.sin(a)
    x, z = t * np.cos(tilt) - p * np.sin(tilt), t * np.sin(tilt) + p * np.cos(tilt)
    if slab:
        x[-slab:], q[-slab:] = rs.uniform(-250, 250, (2, slab))
        z[-slab:] = rs.uniform(0.3, 3.7, slab)
    e = np.clip(np.exp(np.log(20) + 0.8 * rs.normal(size=n)), 10, 1000)
    return [np.ascontiguousarray(v) for v in (x, q, z, e)]


# diameter, core radius, tilt, slab: two bins of nearly 100,000 deposits, several of 20,000, one of
# 150,000 whose spheres overflow the table, and a large bin among small ones
SHAPES = {"two bins": (4.0, 1.0, 0.0, 0), "several": (4.0, 6.0, 0.05, 0),
          "overflow": (4.0, 6.0, 0.0, 130_000), "mixed": (4.0, 2.0, 0.2, 40_000)}


@pytest.mark.parametrize("bins", [200, 3000])       # the 8192- and the 4096-slot table
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_large_bins(ctx, shape, precision, bins):
    d, core, tilt, slab = SHAPES[shape]
    t = _track(220_000, tilt, core, slab, 31)
    spec = ("log", bins, 0.01, 1e5)
    ed = po.edges(*spec)
    oc, oy = np.zeros(bins, dtype=np.int64), np.zeros(bins)
    sx = st.oversample_shifts(HL, d, True, 5, 1, N_OS)
    _, _, os_, _ = po.run_job(*t, half_length=HL, sphere_diameter=d, sxsy=sx, edges_arr=ed,
                              zshift="none", counts=oc, yfy=oy, precision=precision)
    old = {k: ctx.get_param(k) for k in ("precision", "grid", "max_helpers")}
    try:
        ctx.set_param("precision", precision)
        for grid, helpers in ((0, 32), (1, 32), (5, 3), (0, 1)):
            ctx.set_param("grid", grid)
            ctx.set_param("max_helpers", helpers)
            ctx.clear()
            hid = ctx.histogram(*spec)
            jid = ctx.submit(*t, half_length=HL, sphere_diameter=d, n_oversamples=N_OS, hist=hid,
                             seed=5, track_id=1, zshift="none")
            ctx.run()
            gc, gy = ctx.read_histogram(hid)
            gs = ctx.stats(jid)
            assert_stats_equal([gs], [os_])
            assert_hist_equal([gc], [gy], [oc], [oy])
            assert gs["binned"] > 0
    finally:
        for k, v in old.items():
            ctx.set_param(k, v)
