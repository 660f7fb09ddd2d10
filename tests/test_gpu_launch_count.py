"""The launches a run reports: one reset, the prepare kernels (two more where a job of the launch may run
with boundary flags), one planner launch for up to 64 jobs and the fused kernel, for every launch
group of a pipelined batch by what that group holds."""
import numpy as np
import pytest

import supertrack_b200 as st

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pipeline_bytes,launches", [(0, 1 + 6 + 1 + 1), (400_000, 4 * 7 + 2)])
def test_reported_launches(pipeline_bytes, launches):
    rs = np.random.default_rng(2)
    sizes = [9000] + [1000] * 20      # the first qualifies for windows; groups of 1, 7, 10 and 3 jobs
    with st.Context(0) as c:
        c.set_param("pipeline_bytes", pipeline_bytes)
        hid = c.histogram("log", 200, 0.01, 1e4)
        tracks = [np.concatenate([rs.normal(size=(2, n)), rs.uniform(-300, 300, (1, n)),
                                  rs.uniform(10, 100, (1, n))]) for n in sizes]
        for j, t in enumerate(tracks):
            c.submit(*[np.ascontiguousarray(a) for a in t], half_length=300.0, sphere_diameter=1.0,
                     n_oversamples=4, hist=hid, seed=1, track_id=j)
        c.enable_timing(True)
        c.run()
        assert c.last_timing()[2] == launches
