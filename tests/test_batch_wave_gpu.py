"""Batches at the totals where the walk begins to fill the GPU (768 threads an SM, 116,736 on 152 SMs): a
run equals the same substeps with an event between any two passes, bit for bit."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def scene(n, seed):
    side = int(np.ceil(n ** (1.0 / 3.0)))
    w = W.dam_break(dims=(side,) * 3, spacing=0.02, map_res=24, jitter=0.2, seed=seed)
    vel = np.random.default_rng(seed).standard_normal((n, 3)).astype(np.float32)
    return replace(w, pos=w.pos[:n].copy(), vel=vel, sph=replace(w.sph, n_particles=n))


@pytest.mark.parametrize("total", [70_001, 116_735, 116_736, 160_001])
def test_run_equals_substeps_with_events_between(total):
    sizes = [2048, 9001, 20_000, 33_333]
    scenes = [scene(n, k) for k, n in enumerate(sizes + [total - sum(sizes)])]
    a, b = W.build_batch(scenes), W.build_batch(scenes)
    a.substeps(8)
    b.profile_substeps(8)
    for s in range(len(scenes)):
        for x, y in zip(a.get_neighbor_arrays(s), b.get_neighbor_arrays(s)):
            assert np.array_equal(x, y), s
        sa, sb = a.copy_data_buffers(s), b.copy_data_buffers(s)
        for k in sa:
            assert np.array_equal(sa[k], sb[k]), (s, k)
