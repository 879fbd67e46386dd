"""Skin lists just below, at and just above their capacity of 96 candidates, so that fills end inside a
list's last quad and some particles beside listed ones are walked: sums and neighbour sets against the
bucket walk (tests/test_list_build_gpu.py's bar)."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_list_build_gpu import H, compare, scene

pytestmark = pytest.mark.gpu
spatial = pytest.importorskip("scipy.spatial")


@pytest.mark.parametrize("spacing", [0.0146, 0.01478, 0.015])
def test_lists_about_their_capacity(spacing):
    w = scene(50_653, spacing, H, (0.3, 0.1, 0.2), seed=2)
    x = w.pos[:: 17].astype(np.float64)
    near = spatial.cKDTree(w.pos.astype(np.float64)).query_ball_point(x, 1.05 * H, return_length=True)
    assert all(np.any(near == k) for k in (93, 94, 95, 96, 97))
    compare(w)
