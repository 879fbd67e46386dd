"""The walk-staging value is stored for programs that set it, off by default, and a tuning file's value,
whatever it is, leaves the walk of a dense crowd as it is."""
from __future__ import annotations

import numpy as np
import pytest

from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_value_is_off_by_default_and_kept():
    w = W.dam_break(dims=(8, 8, 8), map_res=0)
    m, b = W.build_model(w), W.build_batch([w, w])
    for x in (m, b):
        assert x.get_tune_config()["walk_staging"] == 0
        x.set_walk_staging(True)
        assert x.get_tune_config()["walk_staging"] == 1
        x.set_tune_config(walk_staging=0)
        assert x.get_tune_config()["walk_staging"] == 0


@pytest.mark.parametrize("value", [0, 1])
def test_crowd_is_walked_the_same_for_either_value(value):
    w = W.stress_4m(n_uniform=100_000, n_blob=30_000, map_res=0)
    a, b = W.build_model(w), W.build_model(w)
    a.set_walk_staging(value)
    b.set_skin(0.0)
    for m in (a, b):
        m.set_neighbor_capacity(640)
        m.substeps(1)
    sa, sb = a.copy_data_buffers(), b.copy_data_buffers()
    for k in sa:
        assert np.array_equal(sa[k], sb[k]), k
