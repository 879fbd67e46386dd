"""Neighbour lists at capacities around a whole quad of entries: lists that end anywhere in their
last quad, or overflow it, give the steps of a capacity no list reaches, bit for bit, whichever pass
wrote them (three lanes per particle, the walk, the skin lists, a batch)."""
from __future__ import annotations

import numpy as np
import pytest

import vkfluidsim_gb300 as vfs
from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu

H = 0.04


def scene(n, seed):
    side = int(np.ceil(n ** (1.0 / 3.0)))
    w = W.dam_break(dims=(side,) * 3, spacing=0.02, box=(1e3,) * 3, map_res=0, jitter=0.3, seed=seed)
    w.sim = vfs.SimulationParameters((0.0, 0.0, -9.81), H)
    w.pos = np.ascontiguousarray(w.pos[:n])
    w.vel = np.zeros_like(w.pos)
    return w


@pytest.mark.parametrize("slots", [29, 30, 31, 32, 33])
@pytest.mark.parametrize("n, skin", [(20_000, 0.05), (42_875, 0.05), (42_875, 0.0), (70_001, 0.05)])
def test_capacities_around_a_quad(n, skin, slots):
    # ~32 in-range neighbours: a good part of the lists overflow at each of these capacities.
    w = scene(n, seed=n)
    few, many = W.build_model(w), W.build_model(w)
    for m, c in ((few, slots), (many, 512)):
        m.set_skin(skin)
        m.set_neighbor_capacity(c)
        m.substeps(2)
    a, b = few.copy_data_buffers(), many.copy_data_buffers()
    for k in b:
        assert np.array_equal(a[k], b[k]), k
