"""The particles of a batch whose lists are unusable (small tables whose keys collide) beside scenes
that sum theirs: walked a warp per particle, a thread per particle in a longer queue, and without
any lists, the first substep is the same bit for bit."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def scene(n, seed):
    side = int(np.ceil(n ** (1.0 / 3.0)))
    w = W.dam_break(dims=(side,) * 3, spacing=0.02, map_res=24, jitter=0.2, seed=seed)
    return replace(w, pos=w.pos[:n].copy(), vel=w.vel[:n].copy(), sph=replace(w.sph, n_particles=n))


@pytest.mark.parametrize("small", [1, 4, 5, 9])  # walkers: 3,400 each; the line is 16,384
def test_colliding_scenes_beside_listed_ones(small):
    scenes = [scene(40_000, 1)] + [scene(3400, 2 + k) for k in range(small)]
    lists, walk = W.build_batch(scenes), W.build_batch(scenes)
    walk.set_skin(0.0)
    for b in (lists, walk):
        b.substeps(1)
    assert lists.skin_builds(0) == 1
    for s in range(len(scenes)):
        for x, y in zip(lists.get_neighbor_arrays(s), walk.get_neighbor_arrays(s)):
            assert np.array_equal(x, y), s
        a, c = lists.copy_data_buffers(s), walk.copy_data_buffers(s)
        for k in a:
            assert np.array_equal(a[k], c[k]), (s, k)
