"""The tuner leaves alone what a model of its size does not run: the radix passes and the cell-range kernel
up to 65,536 particles (sorted in one launch), the density pass's shape where three lanes share a
particle."""
from __future__ import annotations

from dataclasses import replace

import pytest

from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SORT = dict(sort_digit_bits=5, sort_tile_items=12, cell_block=128)
SHAPE = dict(nbr_block=64, nbr_min_blocks=12)


@pytest.mark.parametrize("n, kept", [(4096, {**SORT, **SHAPE}), (65_536, SORT), (65_537, {})])
def test_unused_choices_stay(n, kept):
    w = W.dam_break(dims=(41,) * 3, spacing=0.02, map_res=0, jitter=0.2)
    w = replace(w, pos=w.pos[:n].copy(), vel=w.vel[:n].copy(), sph=replace(w.sph, n_particles=n))
    m = W.build_model(w)
    m.set_tune_config(**SORT, **SHAPE)
    chosen = m.autotune(repeats=1, use_cache=False)
    assert chosen == m.get_tune_config()
    for k, v in kept.items():
        assert chosen[k] == v, k
    if not kept:  # (the tuner tries 6, 7 and 8 bits)
        assert chosen["sort_digit_bits"] != SORT["sort_digit_bits"]
    m.substeps(2)
