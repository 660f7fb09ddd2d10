"""The planner at the sizes where its launches change (one CTA plans the batch; it writes the items of
up to 64 jobs itself, a second launch those of larger batches; jobs beyond 1,024 take another round
of its threads), the same jobs run twice (the second time from a CUDA graph), and the call without
allocation at the sizes where its spill tables change. Counts bit-exact against the CPU oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

import pyoracle as po
import supertrack_b200 as st
from supertrack_b200 import _capi

pytestmark = pytest.mark.gpu

HL, D, SPEC, SEED = 100.0, 5.0, ("log", 100, 0.01, 1e4), 3


def _track(n, seed):
    rs = np.random.default_rng(seed)
    p = np.cumsum(rs.normal(size=(n, 3)) * 1.5, axis=0) + rs.normal(size=3) * 20
    p = np.ascontiguousarray(np.clip(p, -90, 90).T)
    return [*p, rs.uniform(10, 1000, n)]


def _oracle(t, track_id, n_os, counts, yfy):
    sx = st.oversample_shifts(HL, D, True, SEED, track_id, n_os)
    po.run_job(*t, half_length=HL, sphere_diameter=D, sxsy=sx, edges_arr=po.edges(*SPEC),
               zshift="none", counts=counts, yfy=yfy)


@pytest.mark.parametrize("n_jobs", [1, 63, 64, 65, 1024, 1025])
def test_batches_around_the_planner_sizes(ctx, n_jobs):
    rs = np.random.default_rng(n_jobs)
    ctx.clear()
    hid = ctx.histogram(*SPEC)
    counts, yfy = np.zeros(100, dtype=np.int64), np.zeros(100)
    for j in range(n_jobs):
        t, n_os = _track(int(rs.integers(0, 200)), j), int(rs.integers(0, 5))
        ctx.submit(*t, half_length=HL, sphere_diameter=D, n_oversamples=n_os, hist=hid, seed=SEED,
                   track_id=j, zshift="none")
        _oracle(t, j, n_os, counts, yfy)
    for rerun in range(3):
        ctx.reset_histogram(hid)
        ctx.jobs_reset()
        ctx.run()
        got, gy = ctx.read_histogram(hid)
        assert np.array_equal(got, counts)
        np.testing.assert_allclose(gy, yfy, rtol=1e-12, atol=0)


@pytest.mark.parametrize("n", [0, 1, 511, 512, 513, 2048, 2049, 4096, 4097, 8193, 16384])
def test_call_without_allocation_around_its_table_sizes(n):
    t, n_os = _track(n, n), 40
    dev = [torch.tensor(a, device="cuda", dtype=torch.float64) for a in t]
    counts = torch.zeros(100, dtype=torch.int64, device="cuda")
    yfy = torch.zeros(100, dtype=torch.float64, device="cuda")
    v, d = _capi.st_track_view(), _capi.st_job_desc()
    v.x, v.y, v.z, v.edep = [a.data_ptr() for a in dev]
    v.n, v.on_device = n, 1
    d.half_length, d.sphere_diameter, d.zshift, d.shift_track = HL, D, st.ZSHIFT["none"], 1
    d.n_oversamples, d.hist_id, d.seed, d.track_id = n_os, -1, SEED, 7
    torch.cuda.synchronize()
    rc = _capi.lib().st_superimpose_noalloc(C.byref(v), C.byref(d), st.HIST_TYPES["log"], 100,
                                            SPEC[2], SPEC[3], counts.data_ptr(), yfy.data_ptr(),
                                            None, None)
    assert rc == _capi.ST_OK
    oc, oy = np.zeros(100, dtype=np.int64), np.zeros(100)
    _oracle(t, 7, n_os, oc, oy)
    assert np.array_equal(counts.cpu().numpy(), oc)
    # the oracle adds the values of a bin (all positive) one by one: one rounding per addition
    np.testing.assert_allclose(yfy.cpu().numpy(), oy, rtol=max(n * n_os, 1) * 2.0 ** -52, atol=0)
