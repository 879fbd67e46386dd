"""The one-launch sort of a small batch: every scene's keys, permutation and offsets, whose keys start at the
scene's own, equal those of a model of the scene alone, bit for bit, and its state too."""
from __future__ import annotations

import numpy as np
import pytest

from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [[(19, 17, 23), (11, 13, 9)], [(1, 1, 1), (32, 32, 32), (5, 1, 1)],
                                  [(31, 31, 31), (32, 31, 31), (17, 16, 18)]])  # 8,716; 32,774; 65,439 in all
def test_every_scene_of_a_small_batch(dims):
    scenes = [W.dam_break(dims=d, map_res=16, jitter=0.3, seed=k) for k, d in enumerate(dims)]
    b = W.build_batch(scenes)
    for step in range(2):
        b.substeps(1)
        for s, w in enumerate(scenes):
            m = W.build_model(w)
            m.substeps(step + 1)
            for x, y in zip(b.get_neighbor_arrays(s), m.get_neighbor_arrays()):
                assert np.array_equal(x, y), (step, s)
            if sum(v.n for v in scenes) <= 38_912:  # the same density pass (three lanes a particle) in both
                sb, sm = b.copy_data_buffers(s), m.copy_data_buffers()
                for k in sm:
                    assert np.array_equal(sb[k], sm[k]), (step, s, k)
