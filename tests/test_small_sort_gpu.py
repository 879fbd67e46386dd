"""The one-launch sort of small models (keys, stable sort, cell starts in one cluster): sorted keys,
permutation and spatial offsets against a NumPy restatement, bit for bit, at the edges of its
blocks, warps and digit counts, and on both sides of its largest size."""
from __future__ import annotations

import numpy as np
import pytest

import vkfluidsim_gb300 as vfs
from vkfluidsim_gb300 import workloads as W

pytestmark = pytest.mark.gpu
M = np.uint64(0xFFFFFFFF)


def keys_of(x, h, n):
    """HashCell3D(floor(x / h)) % n (spatial_hash_3d.slang:16-32) in float32 and uint32 arithmetic."""
    c = np.floor(x.astype(np.float32) / np.float32(h)).astype(np.int64)
    u = (c + 25).astype(np.uint64) & M
    loc, blk = u % np.uint64(50), u // np.uint64(50)
    bh = (blk[:, 0] * np.uint64(15823) + blk[:, 1] * np.uint64(9737333) + blk[:, 2] * np.uint64(440817757)) & M
    hsh = (loc[:, 0] + np.uint64(50) * (loc[:, 1] + np.uint64(50) * loc[:, 2]) + bh) & M
    return (hsh % np.uint64(n)).astype(np.uint32)


def check(m, x, h):
    """One substep from positions x (slot order): its neighbour arrays against NumPy."""
    n = len(x)
    m.substeps(1)
    keys, perm, offs = m.get_neighbor_arrays()
    k = keys_of(x, h, n)
    order = np.argsort(k, kind="stable").astype(np.uint32)
    want = np.full(n, n, np.uint32)
    first = np.unique(k[order], return_index=True)
    want[first[0]] = first[1]
    assert np.array_equal(keys, k[order]) and np.array_equal(perm, order) and np.array_equal(offs, want)


def model(x, h=0.04):
    sim = vfs.SimulationParameters((0.0, 0.0, -9.81), h)
    sph = vfs.SPHParameters(1.0, 1, len(x), 2e-4, 1000.0, (1e3,) * 3, (-500.0,) * 3)
    m = vfs.WCSPHWithBoundaryModel(sim, sph, vfs.WCSPHParameters(1e4, 50.0, 7.0, 0.001))
    rng = np.random.default_rng(len(x))
    m.set_particle_state(x, (rng.random(x.shape).astype(np.float32) - 0.5) * 20.0)
    return m


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 255, 256, 257, 1023, 1025, 4097, 8191, 8192, 8193,
                               16384, 16385, 32767, 32769, 40001, 65535, 65536, 65537])
def test_sizes(n):
    rng = np.random.default_rng(n)
    side = 0.02 * n ** (1.0 / 3.0)
    x = ((rng.random((n, 3)) - 0.3) * side).astype(np.float32)  # negative cells too
    m = model(x)
    check(m, x, m.get_parameters()[0].smooth_radius)
    check(m, m.copy_data_buffers()["positions"], m.get_parameters()[0].smooth_radius)


@pytest.mark.parametrize("kind", ["one cell", "few cells", "sparse"])
def test_distributions(kind):
    rng = np.random.default_rng(7)
    n = 5000
    if kind == "one cell":
        x = (rng.random((n, 3)) * 0.039).astype(np.float32)
    elif kind == "few cells":
        x = (rng.integers(0, 3, (n, 3)) * 0.3 + rng.random((n, 3)) * 0.03).astype(np.float32)
    else:
        x = ((rng.random((n, 3)) - 0.5) * 400.0).astype(np.float32)
    m = model(x)
    check(m, x, m.get_parameters()[0].smooth_radius)


def test_host_round_trip_and_batch_agree_with_the_model():
    """The host round trip's sort reads the page-locked positions itself; a batch's keys carry scene
    offsets: both equal the plain model's substep bit for bit."""
    torch = pytest.importorskip("torch")
    w = W.dam_break(dims=(19, 17, 23), map_res=16, seed=3)
    plain, host = W.build_model(w), W.build_model(w)
    plain.substeps(1)
    pin = [torch.empty(a.shape, dtype=torch.float32, pin_memory=True) for a in (w.pos, w.vel)]
    for t, a in zip(pin, (w.pos, w.vel)):
        t.copy_(torch.from_numpy(a))
    out = {k: torch.empty(s, dtype=torch.float32, pin_memory=True).numpy()
           for k, s in (("positions", (w.n, 3)), ("velocities", (w.n, 3)), ("densities", (w.n,)))}
    got = host.step_host(pin[0].numpy(), pin[1].numpy(), 1, out)
    ref = plain.copy_data_buffers()
    for k in ref:
        assert np.array_equal(got[k], ref[k]), k
    for a, b in zip(plain.get_neighbor_arrays(), host.get_neighbor_arrays()):
        assert np.array_equal(a, b)
    b = W.build_batch([w, W.dam_break(dims=(11, 13, 9), map_res=16, seed=4)])
    b.substeps(1)
    for a, c in zip(plain.get_neighbor_arrays(), b.get_neighbor_arrays(0)):
        assert np.array_equal(a, c)
