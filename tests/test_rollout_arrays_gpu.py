"""After a rollout's forward and backward passes the model holds its own sorted arrays: the last
substep's, as plain stepping leaves them, also once the rollout is gone."""
from __future__ import annotations

import gc
from dataclasses import replace

import numpy as np
import pytest

from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, steps, every", [(2000, 5, 2), (65_536, 4, 4), (70_001, 3, 2)])
def test_neighbour_arrays_after_a_rollout(n, steps, every):
    from vkfluidsim_gb300.adjoint import Rollout

    side = int(np.ceil(n ** (1.0 / 3.0)))
    w = W.dam_break(dims=(side,) * 3, spacing=0.0275, map_res=0, jitter=0.2, seed=n, box=(5.0,) * 3)
    w = replace(w, pos=w.pos[:n].copy(), vel=w.vel[:n].copy(), sph=replace(w.sph, n_particles=n))
    plain, m = W.build_model(w), W.build_model(w)
    for x in (plain, m):  # (a rollout alone does not make the arrays of a fresh model readable)
        x.substeps(1)
    plain.substeps(steps)
    ro = Rollout(m, steps, every)
    ro.forward()
    for x, y in zip(plain.get_neighbor_arrays(), m.get_neighbor_arrays()):
        assert np.array_equal(x, y)
    ro.backward(np.ones((n, 3), np.float32))
    del ro
    gc.collect()
    keys, perm, _ = m.get_neighbor_arrays()
    assert np.array_equal(np.sort(perm), np.arange(n, dtype=np.uint32))
    assert np.all(np.diff(keys.astype(np.int64)) >= 0)
