"""A batch sums its scenes' skin lists only where they hold enough particles (98,304) or leave few to walk
(16,384): on both sides of either line its scenes hold the parity bar against the same batch without
lists, with the same neighbour arrays."""
from __future__ import annotations

import numpy as np
import pytest

from tests.helpers import RTOL, normwise_rel
from tests.test_batch_walkers_gpu import scene
from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("listed", [40_000, 98_303, 98_304])
@pytest.mark.parametrize("small", [4, 5])  # scenes of 3,400 whose keys collide: 13,600 and 17,000 walkers
def test_lists_and_walkers_of_a_batch(listed, small):
    scenes = [scene(listed, 1)] + [scene(3400, 2 + k) for k in range(small)]
    lists, walk = W.build_batch(scenes), W.build_batch(scenes)
    walk.set_skin(0.0)
    for step in range(4):
        for b in (lists, walk):
            b.substeps(1)
        for s in range(len(scenes)):
            for x, y in zip(lists.get_neighbor_arrays(s), walk.get_neighbor_arrays(s)):
                assert np.array_equal(x, y), (step, s)
            a, c = lists.copy_data_buffers(s), walk.copy_data_buffers(s)
            for k in a:
                assert normwise_rel(a[k], c[k]) <= RTOL, (step, s, k)
    assert lists.skin_builds(0) == 1
