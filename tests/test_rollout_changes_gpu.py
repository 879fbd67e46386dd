"""A rollout used again after its model changed: the gradients are those of a rollout created then.
Full segments before the last replay a recorded graph (12 substeps in segments of 5: two of them),
which holds the parameters, buffers and objects of the time it was recorded. Bar: 1e-5 relative, as
for repeated gradients (atomic summation order)."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

import vkfluidsim_gb300 as vfs
from tests import adjoint_scene as S
from tests.helpers import normwise_rel
from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-5


def gradients(ro, w):
    ro.model.set_particle_state(w.pos, w.vel)
    ro.forward()
    x = ro.final_positions_by_id()
    return x, ro.backward((w.pos - w.pos.mean(axis=0) + w.vel).astype(np.float32))


def sort_config(m, w):
    m.set_tune_config(sort_digit_bits=6, sort_tile_items=8)


def objects(m, w):
    for k in range(3):
        m.add_analytic_object(vfs.AnalyticObject(vfs.SHAPE_SPHERE, (0.05,), position=(0.05 + 0.1 * k, 0.42, 0.15),
                                                 resolution=(16,) * 3))


def big_scene():
    """70,000 particles: more than the one-launch sort takes, so the sort's scratch is in use."""
    w = W.dam_break(dims=(50, 40, 35), spacing=0.019, box=(2.0, 2.0, 2.0), map_res=24, stiffness=20.0,
                    viscosity=0.02, seed=7, dt=1e-4)
    return replace(w, sim=replace(w.sim, smooth_radius=0.04), vel=vfs.generate_fourier_velocity(w.pos, 8, 0.5, 11))


CHANGES = {
    "viscosity and stiffness": (S.scene, lambda m, w: m.set_parameters(
        wcsph=replace(w.wcsph, viscosity_strenght=0.5 * w.wcsph.viscosity_strenght,
                      stiffness=0.5 * w.wcsph.stiffness))),
    "time step": (S.scene, lambda m, w: m.set_parameters(sph=replace(w.sph, fixed_dt=2.0 * w.sph.fixed_dt))),
    "boundary objects": (S.scene, objects),
    "sort configuration": (big_scene, sort_config),
}


@pytest.mark.parametrize("change", sorted(CHANGES))
def test_gradients_follow_a_change_of_the_model(change):
    from vkfluidsim_gb300.adjoint import Rollout

    make, apply = CHANGES[change]
    w = make()
    m = W.build_model(w)
    m.set_skin(0.0)  # lists sum in the order of their last build, which is not the same in two runs
    ro = Rollout(m, S.STEPS, S.EVERY)
    gradients(ro, w)
    apply(m, w)
    x, g = gradients(ro, w)
    x_new, want = gradients(Rollout(m, S.STEPS, S.EVERY), w)
    assert np.array_equal(x, x_new)
    for k in ("dnu", "dk"):
        assert abs(g[k] - want[k]) <= TOL * abs(want[k]), k
    for k in ("dv0", "dx0"):
        assert normwise_rel(g[k], want[k]) <= TOL, k


def test_a_changed_neighbour_capacity_is_refused_in_every_segment():
    """The records have the capacity of the rollout's creation; a backward pass whose segments are
    all replayed refuses another one too."""
    from vkfluidsim_gb300.adjoint import Rollout

    w = S.scene()
    m = W.build_model(w)
    ro = Rollout(m, 2 * S.EVERY, S.EVERY)
    seed = gradients(ro, w)[0]
    m.set_neighbor_capacity(64)
    for call in (lambda: ro.backward(seed), ro.forward):
        with pytest.raises(vfs.VfsError):
            call()
