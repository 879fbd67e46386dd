"""The kernels of a substep and of a pair sort are launched so that each may become resident before
the one ahead of it ends. The same work with an event between any two phases (profile_substeps),
and a captured sort replayed on new keys, give the same bits."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

from vkfluidsim_gb300 import primitives
from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("side, fast", [(6, 0.0), (31, 0.5), (37, 0.5), (45, 3.0), (68, 3.0)])
def test_substeps_equal_substeps_with_events_between(side, fast):
    w = W.dam_break(dims=(side,) * 3, spacing=0.02, box=(side * 0.03,) * 3, map_res=0, jitter=0.3, seed=side)
    w.vel = (np.random.default_rng(side).standard_normal(w.pos.shape) * fast).astype(np.float32)
    a, b = W.build_model(w), W.build_model(w)
    a.substeps(12)
    b.profile_substeps(12)
    for x, y in zip(a.get_neighbor_arrays(), b.get_neighbor_arrays()):
        assert np.array_equal(x, y)
    sa, sb = a.copy_data_buffers(), b.copy_data_buffers()
    for k in sa:
        assert np.array_equal(sa[k], sb[k]), k


@pytest.mark.parametrize("side", [12, 36])
def test_runs_equal_single_substeps(side):
    """Runs replay graphs of four substeps and the rest one by one; a parameter change in between
    captures both again."""
    w = W.dam_break(dims=(side,) * 3, spacing=0.02, box=(side * 0.03,) * 3, map_res=0, jitter=0.3, seed=side)
    a, b = W.build_model(w), W.build_model(w)
    for count in (1, 3, 4, 5, 11):
        a.substeps(count)
        for _ in range(count):
            b.substeps(1)
        for m in (a, b):
            m.set_parameters(wcsph=replace(w.wcsph, stiffness=40.0 + count))
    sa, sb = a.copy_data_buffers(), b.copy_data_buffers()
    for k in sa:
        assert np.array_equal(sa[k], sb[k]), k


@pytest.mark.parametrize("n", [1000, 70_001, 1_000_000])
def test_captured_sort_replays(n):
    keys = torch.empty(n, dtype=torch.int32, device="cuda")
    items = torch.empty(n, dtype=torch.int32, device="cuda")
    keys.random_(0, n)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        primitives.sort_pairs(items.data_ptr(), keys.data_ptr(), n, n - 1, s.cuda_stream)
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        primitives.sort_pairs(items.data_ptr(), keys.data_ptr(), n, n - 1, s.cuda_stream)
    for seed in (1, 2):
        fresh = torch.from_numpy(np.random.default_rng(seed).integers(0, n, n).astype(np.int32)).cuda()
        keys.copy_(fresh)
        items.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        want, perm = torch.sort(fresh, stable=True)
        assert torch.equal(keys, want)
        assert torch.equal(items, perm.to(torch.int32))
    assert primitives.sort_status() == 0
