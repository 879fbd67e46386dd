"""A run of substeps whose state is put back to its beginning each time, and whose skin lists die shortly
before its end: from a few runs on the lists stem from its middle and no run builds any. States that never
come back cost at most a build at each end of a run, and a few tries. Drifting lattices (one velocity, no
gravity, below rest density), of the sizes that rebuild in the next substep and at once."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

from tests.helpers import RTOL, normwise_rel
from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class DeviceArray:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n, 4), "typestr": "<f4", "data": (ptr, False), "version": 3}


def drifting(side):
    w = W.dam_break(dims=(side,) * 3, spacing=0.02, box=(side * 0.04,) * 3, map_res=0)
    w.pos = (w.pos + np.float32(0.2)).astype(np.float32)
    w.sim = replace(w.sim, gravity=(0.0, 0.0, 0.0))
    w.vel = np.zeros_like(w.pos)
    w.vel[:, 0] = 0.8  # 1.6e-4 a substep: h skin / 2 = 1e-3 is six of them
    return w


def putter(w, m):
    p, v = (torch.as_tensor(DeviceArray(a, w.n), device="cuda") for a in m.device_state())
    ids = torch.arange(w.n, device="cuda", dtype=torch.int32).view(torch.float32)
    pos = torch.cat([torch.from_numpy(w.pos).cuda(), ids[:, None]], 1)
    vel = torch.cat([torch.from_numpy(w.vel).cuda(), torch.zeros(w.n, 1, device="cuda")], 1)

    def put(shift=0.0):
        m.synchronize()
        p.copy_(pos)
        p[:, 0] += shift
        v.copy_(vel)
        torch.cuda.synchronize()

    return put


@pytest.mark.parametrize("side", [36, 65])
@pytest.mark.parametrize("run", [8, 10, 13])
def test_runs_put_back_to_one_state_keep_their_lists(side, run):
    w = drifting(side)
    m, walk = W.build_model(w), W.build_model(w)
    walk.set_skin(0.0)
    put, put_walk = putter(w, m), putter(w, walk)
    builds = []
    for _ in range(24):
        put()
        m.substeps(run)
        builds.append(m.skin_builds())
    assert builds[-1] == builds[11], builds
    put_walk()
    walk.substeps(run)
    for x, y in zip(m.get_neighbor_arrays(), walk.get_neighbor_arrays()):
        assert np.array_equal(x, y)
    a, b = m.copy_data_buffers(), walk.copy_data_buffers()
    for k in a:
        assert normwise_rel(a[k], b[k]) <= RTOL, k


@pytest.mark.parametrize("side", [36, 65])
def test_runs_of_ever_new_states_do_not_try_often(side):
    w = drifting(side)
    m = W.build_model(w)
    put = putter(w, m)
    for k in range(40):
        put(0.01 * k)
        m.substeps(8)
    assert m.skin_builds() <= 2 * 40 + 6
