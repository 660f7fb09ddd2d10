"""Exact sums in the fused kernel's shared memory, word by word: every deposit of a track in the
same few spheres (each 32-bit word of a sum takes many carries, from many warps at once), and
every sphere in the same histogram bin. Sphere energies, counts and hits are compared with the
CPU oracle bit for bit, y*f(y) within the rounding of the oracle's own running sums."""
import numpy as np
import pytest

import pyoracle as po
import supertrack_b200 as st

pytestmark = pytest.mark.gpu

# per-sphere energy ranges: 45 bits between the smallest and the largest contribution, both signs
# (a positive and a negative total), all-ones mantissas (a carry out of the low word on nearly every
# addition), and one value for all (every sphere of one hit in one bin)
ENERGIES = {
    "wide": lambda rs, n: np.exp2(rs.uniform(-20, 25, n)),
    "signed": lambda rs, n: np.where(rs.random(n) < 0.5, -1.0, 1.0) * np.exp2(rs.uniform(0, 30, n)),
    "negative": lambda rs, n: -np.exp2(rs.uniform(0, 8, n)),
    "ones": lambda rs, n: np.nextafter(np.exp2(rs.integers(1, 9, n).astype(float)), 0),
    "equal": lambda rs, n: np.full(n, 17.0),
}


@pytest.mark.parametrize("energies", sorted(ENERGIES))
# (half length, diameter): the one-sphere voxel, a 2^3 lattice of hot spheres, and small spheres
# that take a hit or two each; 3,000 bins run on the 4096-slot table, 200 on the 8192-slot one
@pytest.mark.parametrize("hl,d,bins", [(400.0, 1000.0, 3000), (500.0, 500.0, 200), (100.0, 4.0, 200)])
def test_hot_spheres_and_bins(ctx, energies, hl, d, bins):
    rs = np.random.default_rng(5)
    n, n_os = 20_011, 3
    x, y, z = rs.uniform(-hl / 2, hl / 2, (3, n))
    e = ENERGIES[energies](rs, n)
    spec = ("log", bins, 1e-3, 1e9)
    ctx.clear()
    hid = ctx.histogram(*spec)
    job = ctx.submit(x, y, z, e, half_length=hl, sphere_diameter=d, n_oversamples=n_os, hist=hid,
                     seed=9, zshift="none")
    got = ctx.run_export(n * n_os)
    counts, yfy = ctx.read_histogram(hid)
    stats = ctx.stats(job)
    edges = po.edges(*spec)
    oc, oy = np.zeros(bins, dtype=np.int64), np.zeros(bins)
    sxsy = st.oversample_shifts(hl, d, True, 9, 0, n_os)
    _, _, want, spheres = po.run_job(x, y, z, e, half_length=hl, sphere_diameter=d, sxsy=sxsy,
                                     edges_arr=edges, zshift="none", counts=oc, yfy=oy,
                                     spheres_cap=n * n_os)
    assert (stats["hits"], stats["spheres"], stats["binned"]) == \
        (want["hits"], want["spheres"], want["binned"])
    got = np.sort(got, order=["os", "key"])
    spheres = np.sort(spheres, order=["os", "key"])
    assert np.array_equal(got["key"], spheres["key"]) and np.array_equal(got["y"], spheres["y"])
    assert np.array_equal(counts, oc)
    # the oracle adds a bin's values (all positive) one by one: within one rounding per addition
    np.testing.assert_allclose(yfy, oy, rtol=n * n_os * 2.0 ** -53, atol=0)
