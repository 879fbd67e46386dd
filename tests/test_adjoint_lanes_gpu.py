"""Gradients at the particle counts where the adjoint kernels' split of a neighbour list over lanes
changes, and where the last group or block is partly empty, against the FP64 host adjoint
(tests/fp64_torch_rollout.py). Bar: 1e-3 relative, as for the full-scale rollout."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

import vkfluidsim_gb300 as vfs
from tests.helpers import normwise_rel
from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
pytest.importorskip("scipy")

TOL = 1e-3
STEPS, EVERY = 6, 4


@pytest.mark.parametrize("n", [33, 40959, 40960, 40961, 65535])
def test_gradients_where_the_lane_split_changes(n):
    from tests import fp64_torch_rollout as R
    from vkfluidsim_gb300.adjoint import Rollout

    base = W.dam_break_64k()
    pos = base.pos[:n].copy()
    vel = vfs.generate_fourier_velocity(pos, 8, 0.5, 4)
    w = replace(base, pos=pos, vel=vel, sph=replace(base.sph, n_particles=n))
    ro = Rollout(W.build_model(w), STEPS, EVERY)
    ro.forward()
    # A gradient whose pressure (virial) and viscous (dissipation) sums don't cancel.
    g_x = (pos - pos.mean(axis=0) + vel).astype(np.float32)
    g = ro.backward(g_x)

    def t(v):
        return torch.tensor(float(v), dtype=torch.float64, device="cuda").requires_grad_(True)

    nu, k = t(w.wcsph.viscosity_strenght), t(w.wcsph.stiffness)
    v0 = torch.from_numpy(vel.astype(np.float64)).cuda().requires_grad_(True)
    x = R.rollout(w, nu, k, v0, STEPS, EVERY, grad=True)
    (x * torch.from_numpy(g_x.astype(np.float64)).cuda()).sum().backward()
    assert normwise_rel(g["dv0"], v0.grad.cpu().numpy()) <= TOL
    assert abs(g["dk"] - float(k.grad)) <= TOL * abs(float(k.grad))
    assert abs(g["dnu"] - float(nu.grad)) <= TOL * abs(float(nu.grad))
