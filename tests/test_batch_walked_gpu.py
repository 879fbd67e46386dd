"""A batch of few particles in scenes with lists (three eighths of it, at least 49,152) walks them all where
more than one in six of its particles has no list to sum (scenes of 3,400 whose keys collide), and builds no
more lists; otherwise the moving scene's are rebuilt. The fields hold the parity bar against the batch without lists."""
from __future__ import annotations

import numpy as np
import pytest

from tests.helpers import RTOL, normwise_rel
from tests.test_batch_walkers_gpu import scene
from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large, small, lists_used", [
    (39_999, 2, True), (34_000, 2, True), (33_999, 2, False), (40_000, 4, False), (68_000, 4, True),
    (49_151, 4, False), (49_152, 4, True), (56_000, 28, False), (60_000, 28, True)])
def test_one_walker_in_six(large, small, lists_used):
    scenes = [scene(large, 1)] + [scene(3400, 2 + k) for k in range(small)]
    scenes[0].objects = []  # (the container's map would throw its wall particles)
    scenes[0].pos += np.float32(0.1)
    scenes[0].vel[:, 0] = 0.9
    lists, walk = W.build_batch(scenes), W.build_batch(scenes)
    walk.set_skin(0.0)
    # 1.8e-4 m a substep against h skin / 2 = 1e-3: rebuilt after six, before a colliding scene's wait of
    # eight (to build again) ends.
    for b in (lists, walk):
        b.substeps(8)
    assert (lists.skin_builds(0) > 1) == lists_used
    for s in range(len(scenes)):
        a, c = lists.copy_data_buffers(s), walk.copy_data_buffers(s)
        # (Sorted order may differ where rounding moves a particle over a cell's face.)
        ia, ic = np.argsort(lists.get_ids(s)), np.argsort(walk.get_ids(s))
        for k in a:
            assert normwise_rel(a[k][ia], c[k][ic]) <= 10 * RTOL, (s, k)
