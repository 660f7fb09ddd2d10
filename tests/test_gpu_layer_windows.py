"""Windows of whole z layers against the CPU oracle: hits, spheres, binned spheres and counts
bit-exact, y*f(y) within 1e-12.

The shapes put the window boundaries where they can go wrong: many thin layers per window
(a track along z), layers larger than a window (deposits in a slab, sparse ones whose spheres
overflow the shared table and go through the log, dense ones that stay in it), a track across z
(too many deposits in large layers: it runs with boundary flags instead), lattices with more
layers than bins, deposits on the voxel's faces and on layer boundaries, and just more kept
deposits than the threshold."""
import numpy as np
import pytest

import pyoracle as po
import supertrack_b200 as st
from helpers import assert_hist_equal, assert_stats_equal

pytestmark = pytest.mark.gpu

#: half length, diameter
HL, D = 300.0, 1.0


def _line(rs, n, axis, sigma):
    """n points along an axis through the voxel, in order, with a Gaussian core."""
    p = rs.normal(scale=sigma, size=(n, 3))
    p[:, axis] = np.sort(rs.uniform(-HL, HL, n))
    return p


def _slab(rs, n, side, thick):
    return np.stack([rs.uniform(-side, side, n), rs.uniform(-side, side, n),
                     0.5 * D + rs.uniform(-thick, thick, n)], 1)


def _faces(rs, n):
    """Half of the points on layer boundaries, layer centres and the voxel's faces in z."""
    p = rs.uniform(-HL, HL, (n, 3))
    k = rs.integers(-int(HL), int(HL) + 1, n // 2)
    p[: n // 2, 2] = k * D + rs.choice([0.0, 0.5 * D, 1e-13, -1e-13], n // 2)
    p[:64, 2] = np.nextafter(HL, 0) * rs.choice([-1, 1], 64)
    return p


SHAPES = {
    "along z": lambda rs: (_line(rs, 40_000, 2, 20.0), HL, D),
    "along x": lambda rs: (_line(rs, 60_000, 0, 0.4), HL, D),
    "sparse slab": lambda rs: (np.concatenate([_slab(rs, 30_000, 200.0, 0.4),
                                               _line(rs, 100_000, 2, 40.0)]), HL, D),
    "dense slab": lambda rs: (np.concatenate([_slab(rs, 60_000, 8.0, 0.4),
                                              _line(rs, 200_000, 2, 5.0)]), HL, D),
    "many layers": lambda rs: (_line(rs, 30_000, 2, 2.0), HL, 0.07),
    "faces": lambda rs: (_faces(rs, 20_000), HL, D),
    "threshold": lambda rs: (_line(rs, 16_385, 2, 2.0), HL, D),
}


@pytest.mark.parametrize("bins", [200, 3000])       # the 8192- and the 4096-slot table
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_layer_windows(ctx, shape, precision, bins):
    rs = np.random.default_rng(23)
    p, hl, d = SHAPES[shape](rs)
    x, y, z = [np.ascontiguousarray(p[:, k]) for k in range(3)]
    e = np.clip(np.exp(np.log(20) + 0.8 * rs.normal(size=len(x))), 10, 1000)
    spec, n_os = ("log", bins, 0.01, 1e5), 4
    old = ctx.get_param("precision")
    ctx.set_param("precision", precision)
    try:
        ctx.clear()
        hid = ctx.histogram(*spec)
        jid = ctx.submit(x, y, z, e, half_length=hl, sphere_diameter=d, n_oversamples=n_os,
                         hist=hid, seed=5, track_id=1, zshift="none")
        ctx.run()
        gc, gy = ctx.read_histogram(hid)
        gs = ctx.stats(jid)
    finally:
        ctx.set_param("precision", old)
    ed = po.edges(*spec)
    oc, oy = np.zeros(bins, dtype=np.int64), np.zeros(bins)
    sx = st.oversample_shifts(hl, d, True, 5, 1, n_os)
    _, _, os_, _ = po.run_job(x, y, z, e, half_length=hl, sphere_diameter=d, sxsy=sx,
                              edges_arr=ed, zshift="none", counts=oc, yfy=oy,
                              precision=precision)
    assert_stats_equal([gs], [os_])
    assert_hist_equal([gc], [gy], [oc], [oy])
    assert gs["binned"] > 0
