"""The substep's sort of the particles whose key changed, from none to all of them, at the edges of its
tiles (4,096 keys) and on both sides of the size where its ranking changes (2,097,152 particles): sorted
keys, permutation and spatial offsets against NumPy, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_small_sort_gpu import check, keys_of, model

pytestmark = pytest.mark.gpu

@pytest.mark.parametrize("N, moved", [(100_001, 0), (100_001, 1), (100_001, 4096), (100_001, 4097), (100_001, 100_001),
                                      (2_097_152, 50_000), (2_097_152, 2_097_152), (2_097_153, 50_000),
                                      (2_097_153, 2_097_153)])
def test_counts_of_moved_particles(N, moved):
    rng = np.random.default_rng(1)
    x = ((rng.random((N, 3)) - 0.3) * 0.02 * N ** (1.0 / 3.0)).astype(np.float32)
    m = model(x)
    h = m.get_parameters()[0].smooth_radius
    check(m, x, h)
    # In the order of that sort every key is the slot's previous one; `moved` slots take another's place.
    k = keys_of(x, h, N)
    order = np.argsort(k, kind="stable")
    xs, k = x[order], k[order]
    at = rng.permutation(N)[:moved]
    xs[at] = x[order][(at + N // 2) % N]
    assert np.count_nonzero(keys_of(xs, h, N) != k) == moved
    m.set_particle_state(xs, np.zeros_like(xs))
    check(m, xs, h)
