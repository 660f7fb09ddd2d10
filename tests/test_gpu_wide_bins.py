"""Histograms with a very wide bin: the y*f(y) sum of a bin is kept in shared memory as a 128-bit integer
on the grid of the bin's lower edge, and must not wrap however far above that edge the spheres lie
and however many one CTA collects. Every deposit here is a sphere of its own at its centre, of the
same lineal energy v, so the sum is spheres * v; the tolerance counts the double additions to HBM,
each within 2^-53 of the running sum: one per flush (at least 2^18 - 16,000 deposit*oversamples
apart), or one per sphere where the 128 bits cannot hold the sum."""
import ctypes as C

import numpy as np
import pytest
import torch

import supertrack_b200 as st
from supertrack_b200 import _capi

pytestmark = pytest.mark.gpu

HL, D, N, UPPER = 2500.0, 2.0, 16_000, 1e4


def _track():
    k = np.arange(N)
    z = -HL + D / 2 + D * (k % 2000)
    x = D / 2 + D * (k // 2000)
    return [np.ascontiguousarray(a, dtype=np.float64)
            for a in (x, np.full(N, D / 2), z, np.full(N, 30.0))]


def _check(counts, yfy, n_os, per_sphere):
    spheres = N * n_os
    v = 30.0 / ((2.0 / 3.0) * D)
    assert counts[0] == spheres
    adds = spheres if per_sphere else spheres // (2 ** 18 - N) + 1
    assert abs(yfy[0] - spheres * v) <= spheres * v * (adds + 1) * 2.0 ** -53


# (lower edge, oversamples, sum per sphere in HBM): v is 2^48, 2^61 and 2^104 times the edge; 1e8
# spheres of the first pass 2^127 units of its last place, as few as 2^13 of the second do
CASES = [(1e-13, 10_000, False), (1e-17, 20, True), (1e-30, 3, True)]


@pytest.mark.parametrize("lower,n_os,per_sphere", CASES)
def test_context_on_one_cta(ctx, lower, n_os, per_sphere):
    old = ctx.get_param("grid")
    ctx.set_param("grid", 1)
    try:
        ctx.clear()
        hid = ctx.histogram("lin", 1, lower, UPPER)
        ctx.submit(*_track(), half_length=HL, sphere_diameter=D, n_oversamples=n_os, hist=hid,
                   seed=1, track_id=0, shift_track=False, zshift="none")
        ctx.run()
        counts, yfy = ctx.read_histogram(hid)
    finally:
        ctx.set_param("grid", old)
    _check(counts, yfy, n_os, per_sphere)


@pytest.mark.parametrize("lower,n_os,per_sphere", [(1e-13, 10, False), *CASES[1:]])
def test_call_without_allocation(lower, n_os, per_sphere):
    t = [torch.as_tensor(a, device="cuda") for a in _track()]
    counts = torch.zeros(1, dtype=torch.int64, device="cuda")
    yfy = torch.zeros(1, dtype=torch.float64, device="cuda")
    view, desc, stats = _capi.st_track_view(), _capi.st_job_desc(), _capi.st_job_stats()
    view.x, view.y, view.z, view.edep = [a.data_ptr() for a in t]
    view.n, view.on_device = N, 1
    desc.half_length, desc.sphere_diameter = HL, D
    desc.zshift, desc.shift_track, desc.n_oversamples = st.ZSHIFT["none"], 0, n_os
    desc.seed, desc.track_id, desc.hist_id = 1, 0, -1
    _capi.check(_capi.lib().st_superimpose_noalloc(
        C.byref(view), C.byref(desc), st.HIST_TYPES["lin"], 1, lower, UPPER, counts.data_ptr(),
        yfy.data_ptr(), None, C.byref(stats)), "st_superimpose_noalloc")
    _check(counts.cpu().numpy(), yfy.cpu().numpy(), n_os, per_sphere)
