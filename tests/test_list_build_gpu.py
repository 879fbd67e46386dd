"""The skin-list build (tiles of 32 particles filtered on the tensor cores) and the tiled walk of a
crowd without usable lists: sums and neighbour sets against the per-thread bucket walk, bit for bit,
where the build can go wrong: cells on both sides of hash-block faces on every axis, negative cells,
tables just above the smallest that lists take, runs of keys that pass the table's end, groups of one
to six cells, lists at and over their capacity, isolated particles and particles far outside the
cells' range."""
from __future__ import annotations

import numpy as np
import pytest

import vkfluidsim_gb300 as vfs
from tests.helpers import RTOL, normwise_rel
from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def scene(n, spacing, h, origin=(0.0, 0.0, 0.0), seed=0, jitter=0.2):
    """A jittered cube of n particles from `origin`, no walls."""
    side = int(np.ceil(n ** (1.0 / 3.0)))
    w = W.dam_break(dims=(side,) * 3, spacing=spacing, box=(1e3,) * 3, map_res=0, jitter=jitter, seed=seed)
    w.sim = vfs.SimulationParameters((0.0, 0.0, -9.81), h)
    w.pos = np.ascontiguousarray((w.pos[:n] + np.asarray(origin, np.float32)).astype(np.float32))
    w.vel = np.zeros_like(w.pos)
    return w


def compare(w, slots=128, substeps=3, skin=0.05):
    lists, walk = W.build_model(w), W.build_model(w)
    walk.set_skin(0.0)
    lists.set_skin(skin)
    for m in (lists, walk):
        m.set_neighbor_capacity(slots)
    for s in range(substeps):
        # The first substep builds and sums its lists in the walk's order: bit for bit. Later ones
        # keep the build's order, which is the walk's until neighbours change places: the parity bar.
        lists.substeps(1)
        walk.substeps(1)
        for x, y in zip(lists.get_neighbor_arrays(), walk.get_neighbor_arrays()):
            assert np.array_equal(x, y), f"substep {s + 1}: neighbour arrays"
        a, b = lists.copy_data_buffers(), walk.copy_data_buffers()
        for k in a:
            if s == 0:
                assert np.array_equal(a[k], b[k]), f"substep 1: {k}"
            else:
                assert normwise_rel(a[k], b[k]) <= RTOL, f"substep {s + 1}: {k}"
    assert lists.skin_builds() >= 1 and walk.skin_builds() == 0


H = 0.04


@pytest.mark.parametrize("n, spacing, origin", [
    (42_875, 0.02, (0.0, 0.0, 0.0)),                          # inside one hash block
    (42_875, 0.02, (25 * H - 0.35, 0.0, 0.0)),                # across a block face in x
    (42_875, 0.02, (25 * H - 0.35, 25 * H - 0.31, 25 * H - 0.37)),  # a corner of eight blocks
    (42_875, 0.02, (-25 * H - 0.35, -0.33, -25 * H - 0.3)),   # negative cells, the short block
    (40_001, 0.0185, (0.3, 1.7, -2.9)),                       # a settled fluid, odd size
    (50_653, 0.016, (0.01, 0.02, 0.03)),                      # ~65 within h (1 + skin): lists at capacity
    (39_304, 0.05, (0.0, 0.0, 0.0)),                          # sparse: ~2 neighbours
    (39_304, 0.2, (-3.0, 0.0, 1.0)),                          # isolated particles, no tiles
    (40_000, 0.02, (4.1e3, -7.7e3, 1.3e4)),                   # 300,000 cells out: coarse coordinates
])
def test_built_lists_equal_the_walk(n, spacing, origin):
    compare(scene(n, spacing, H, origin, seed=n))


@pytest.mark.parametrize("skin", [0.001, 0.2, 0.5])
def test_build_at_other_skins(skin):
    compare(scene(42_875, 0.024, H, (0.61, 0.2, 0.93), seed=3), skin=skin)


def test_far_out_and_non_finite_particles():
    """A few particles beyond the range of cell coordinates and a NaN among a normal scene: the
    rest of it is summed as the walk sums it."""
    w = scene(42_875, 0.02, H, (0.0, 0.0, 0.0), seed=5)
    w.pos[17] = (1e12, 0.3, 0.3)
    w.pos[4711] = (-3e11, 1e12, 0.1)
    w.pos[40_000] = (0.31, np.nan, 0.2)
    lists, walk = W.build_model(w), W.build_model(w)
    walk.set_skin(0.0)
    for m in (lists, walk):
        m.substeps(1)
    a, b = lists.copy_data_buffers(), walk.copy_data_buffers()
    for x, y in zip(lists.get_neighbor_arrays(), walk.get_neighbor_arrays()):
        assert np.array_equal(x, y)
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k


@pytest.mark.parametrize("blob, sigma", [(9_000, 0.03), (60_000, 0.06)])
def test_crowd_without_lists_equals_the_walk(blob, sigma):
    """A dense blob (every list over its capacity) in a thin cloud: its particles are a crowd the
    tiles walk (with staging off, a warp per particle)."""
    n = 60_000
    w = W.dam_break(dims=(2, 2, 2), spacing=0.02, box=(2.0, 2.0, 2.0), map_res=0)
    rng = np.random.default_rng(blob)
    x = np.concatenate([rng.random((n, 3)) * 2.0, rng.normal(1.0, sigma, (blob, 3))])
    w.pos = np.clip(x, 0.0, 2.0).astype(np.float32)
    w.vel = np.zeros_like(w.pos)
    w.sim = vfs.SimulationParameters((0.0, 0.0, -9.81), H)
    models = [W.build_model(w) for _ in range(3)]
    models[1].set_walk_staging(False)
    models[2].set_skin(0.0)
    for m in models:
        m.set_neighbor_capacity(512)
        m.substeps(1)
    ref = models[2].copy_data_buffers()
    for m in models[:2]:
        got = m.copy_data_buffers()
        for k in ref:
            assert np.array_equal(got[k], ref[k]), k
