"""A context's first run allocates its arrays; each allocation costs it tens of microseconds and more,
so a qualifying job (windows, boundary flags) must not take more of them than the 26 it needs, and
the run after it none."""
import numpy as np
import pytest
import torch

import supertrack_b200 as st

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
def test_first_run_allocations(precision):
    rs = np.random.default_rng(1)
    t = [torch.as_tensor(a, device="cuda") for a in
         (*rs.normal(scale=5.0, size=(2, 20_000)), np.sort(rs.uniform(-300, 300, 20_000)),
          rs.uniform(10, 1000, 20_000))]
    with st.Context(0) as c:
        c.set_param("precision", precision)
        hid = c.histogram("log", 200, 0.01, 1e4)
        for track in range(2):
            c.clear()
            c.submit(*[a.data_ptr() for a in t], on_device=True, n=20_000, half_length=300.0,
                     sphere_diameter=1.0, n_oversamples=4, hist=hid, seed=1, track_id=track)
            c.run()
            assert c.get_param("last_host_allocs") <= (26 if track == 0 else 0)
