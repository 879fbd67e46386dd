"""A model without lists at the sizes where its walk begins to fill the GPU (768 threads an SM, 116,736
on 152 SMs) and just above the one-launch sort: a run equals the same substeps with an event between
any two passes, bit for bit."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65_537, 116_735, 116_736, 116_737])
def test_run_equals_substeps_with_events_between(n):
    w = W.dam_break(dims=(49,) * 3, spacing=0.02, box=(1.5,) * 3, map_res=0, jitter=0.3, seed=n)
    vel = np.random.default_rng(n).standard_normal((n, 3)).astype(np.float32)
    w = replace(w, pos=w.pos[:n].copy(), vel=vel, sph=replace(w.sph, n_particles=n))
    a, b = W.build_model(w), W.build_model(w)
    for m in (a, b):
        m.set_skin(0.0)
    a.substeps(6)
    b.profile_substeps(6)
    for x, y in zip(a.get_neighbor_arrays(), b.get_neighbor_arrays()):
        assert np.array_equal(x, y)
    sa, sb = a.copy_data_buffers(), b.copy_data_buffers()
    for k in sa:
        assert np.array_equal(sa[k], sb[k]), k
