"""The work a user has this framework do, as cases to measure.

Families (the field ``kind`` of a case):

* ``frame``   a host program's frame loop: the state up from page-locked arrays, the frame's
              substeps, the new state down, in one call (``step_host``).
* ``sim``     a GPU-resident simulation: a checkpoint on the GPU written through ``device_state``,
              a run of substeps, the state read back by particle id without leaving the GPU.
* ``batch``   many independent scenes advanced together (data generation): reset every scene, run,
              read every scene.
* ``adjoint`` a differentiable rollout: forward, then the gradient of a function of the final
              positions with respect to the initial state, viscosity and stiffness.
* ``sort``    the spatial-hash primitives on device buffers: sort the keys, find each cell's start,
              reorder positions and velocities.
* ``view``    one headless picture of a state: particle splat, density grid, raymarch of the grid.

States are jittered lattices, as the benchmark's workloads are: ``ratio`` is the lattice spacing
over the smoothing length (0.5: the benchmark's, below rest density; 0.46: a settled fluid, a
little above it), ``speed`` the amplitude of a smooth velocity field (0: a column that starts to
fall) and ``object`` the boundary object that comes with it. ``exact`` restates the substep in
64 bits from the same inputs.
"""
import math

import numpy as np
import torch

from vkfluidsim_gb300 import (SHAPE_CONTAINER, SHAPE_SPHERE, AnalyticObject, Batch,
                              SimulationParameters, SPHParameters, WCSPHParameters,
                              WCSPHWithBoundaryModel, look_at, perspective, primitives,
                              render_density_raymarch)
from vkfluidsim_gb300.adjoint import Rollout

DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------- cases


def _flow(kind, n, substeps, spacing, ratio=0.46, speed=0.5, dt=2e-4, viscosity=0.01, object="none",
          res=64, sorted=True, skin=0.05, **more):
    return dict(kind=kind, n=n, substeps=substeps, spacing=spacing, ratio=ratio, speed=speed, dt=dt,
                viscosity=viscosity, object=object, res=res, sorted=sorted, skin=skin, **more)


def listed():
    return [
        # The reference's default model: 8,192 particles, 3 iterations a frame, an interactive
        # frame loop. The smallest call, all latency.
        dict(_flow("frame", 8192, 3, 0.02, object="container", res=32), name="frame_8k"),
        # The 32,768-particle dam break of the benchmark, one substep a frame, driven by a host
        # program that keeps its particles in its own order.
        dict(_flow("frame", 32768, 1, 0.02, ratio=0.5, object="container", sorted=False),
             name="frame_32k"),
        # The benchmark's end-to-end leg: the 1M scene up and down the host link every substep.
        dict(_flow("frame", 1048576, 1, 0.0075, ratio=0.5, speed=0.3, dt=1e-4, viscosity=0.001,
                   object="sphere", res=128), name="frame_1m"),
        # A small GPU-resident run, odd size.
        dict(_flow("sim", 5003, 32, 0.02, object="sphere", res=32), name="sim_5k"),
        # A mid-size resident run: more particles than one wave of three-lane work, odd size.
        dict(_flow("sim", 47311, 32, 0.02, object="sphere"), name="sim_47k"),
        # The benchmark's plain leg: the 1M column in its first substeps, starting to fall.
        dict(_flow("sim", 1048576, 16, 0.0075, ratio=0.5, speed=0.0, dt=1e-4, object="sphere",
                   res=128), name="sim_1m_fall"),
        # The same size as a settled fluid in motion around an obstacle.
        dict(_flow("sim", 1048576, 16, 0.0075, dt=1e-4, viscosity=0.001, object="sphere", res=128),
             name="sim_1m_flow"),
        # The benchmark's stress cloud as it is loaded: 4.2M uniform particles and a dense blob of
        # 419k, in no order, with long neighbour lists.
        dict(kind="sim", n=4613734, blob=419430, substeps=1, spacing=0.01, ratio=0.5, speed=0.0,
             dt=1e-4, viscosity=0.01, object="container", res=128, sorted=False, skin=0.05,
             slots=1536, name="stress_4m"),
        # Data generation: 64 dam breaks of uneven size (the benchmark's batch, a quarter of it).
        dict(kind="batch", scenes=64, n_min=2048, n_max=65536, substeps=32, spacing=0.02, ratio=0.5,
             dt=2e-4, res=64, name="batch_64"),
        # Training: the 65,536-particle differentiable rollout, shortened to two segments.
        dict(kind="adjoint", n=65536, substeps=24, every=12, spacing=0.0275, ratio=0.0275 / 0.06,
             speed=0.2, dt=2e-4, viscosity=0.01, object="none", res=0, sorted=True, skin=0.05,
             name="adjoint_64k"),
        # The spatial-hash primitives by themselves, odd size.
        dict(kind="sort", n=1000003, name="sort_1m"),
        # A picture of the 1M scene.
        dict(_flow("view", 1048576, 0, 0.0075, width=1280, height=720, grid=128), name="view_1m"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "sim", "sim", "sim", "sim", "batch", "adjoint", "sort", "view"])
    ratio = round(rng.uniform(0.45, 0.55), 4)
    speed = rng.choice([0.0, round(rng.uniform(0.05, 1.0), 3)])
    sort = rng.random() < 0.6
    if kind == "sort":
        return dict(kind="sort", n=_log_int(rng, 1000, 4000000))
    if kind == "batch":
        n_min = _log_int(rng, 1500, 4000)
        return dict(kind="batch", scenes=_log_int(rng, 3, 48), n_min=n_min,
                    n_max=_log_int(rng, 8 * n_min, 16 * n_min), substeps=rng.randrange(8, 33),
                    spacing=0.02, ratio=ratio, dt=2e-4, res=rng.choice([24, 32, 48]))
    if kind == "adjoint":
        every = rng.randrange(4, 11)
        return dict(kind="adjoint", n=_log_int(rng, 4000, 60000), substeps=every + rng.randrange(1, every + 1),
                    every=every, spacing=0.0275, ratio=ratio, speed=speed, dt=2e-4, viscosity=0.01,
                    object=rng.choice(["none", "sphere"]), res=32, sorted=sort, skin=0.05)
    n = _log_int(rng, 2000, 1000000)
    spacing = 0.02 if n < 200000 else 0.0075
    dt, visc = (2e-4, 0.01) if n < 200000 else (1e-4, 0.001)
    obj = rng.choice(["none", "sphere", "container"])
    skin = rng.choice([0.05, 0.05, 0.0, round(rng.uniform(0.02, 0.15), 3)])
    if kind == "view":
        return dict(_flow("view", n, 0, spacing, ratio, speed, width=rng.randrange(301, 1280),
                          height=rng.randrange(201, 720), grid=rng.randrange(33, 128)))
    if kind == "frame":
        # Several substeps a frame are an interactive program's; those stay small.
        return _flow("frame", n, 1 if n > 60000 else rng.choice([1, 2, 3]), spacing, ratio, speed, dt,
                     visc, obj, rng.choice([32, 48, 64]), sort, skin)
    return _flow("sim", n, rng.randrange(4, 17), spacing, ratio, speed, dt, visc, obj,
                 rng.choice([32, 48, 64]), sort, skin, slots=rng.choice([128, 128, 64, 200]))


# ---------------------------------------------------------------- inputs, from the seed alone


def _f32(x):
    return float(np.float32(x))


def _h(case):
    return _f32(case["spacing"] / case["ratio"])


def _dims(n):
    """A cube, or for a large scene a column twice as long as wide. (A small scene that spans
    several of the hash's blocks counts some neighbours twice, as the reference does, and bursts.)"""
    k = 1 if n < 125000 else 2
    a = max(1, math.ceil((n / k) ** (1.0 / 3.0)))
    return k * a, a, max(1, math.ceil(n / (k * a * a)))


def _geometry(case, n):
    """Extent of the column, its box, and its boundary object (shape, size, centre)."""
    h = _h(case)
    if case.get("blob"):
        box = (4.0, 2.0, 2.0)
        return box, box, (SHAPE_CONTAINER, (2.0, 1.0, 1.0), (2.0, 1.0, 1.0))
    d = _dims(int(1.1 * n) if case["object"] == "sphere" and case["speed"] else n)
    ext = tuple(case["spacing"] * k for k in d)
    box = tuple(_f32(1.5 * e) for e in ext)
    if case["object"] == "container":
        # Half a smoothing length of room all around: a fluid poured against the walls of its
        # volume map would start far above rest density there and burst.
        return ext, box, (SHAPE_CONTAINER, tuple(0.5 * b + 0.5 * h for b in box), tuple(0.5 * b for b in box))
    if case["object"] == "sphere":
        # In the middle of a moving fluid; in front of a column at rest, as in the benchmark.
        r = _f32(max(0.15 * ext[1], 1.5 * h))
        c = tuple(0.5 * e for e in ext) if case["speed"] else (1.5 * ext[0], 0.5 * ext[1], r)
        return ext, box, (SHAPE_SPHERE, (r,), tuple(_f32(x) for x in c))
    return ext, box, None


def _keys(cells, n):
    """The hash key of integer cells (the reference's spatial hash, which is part of its format)."""
    u = (cells + 25) & 0xFFFFFFFF
    loc, blk = u % 50, u // 50
    bh = (blk[..., 0] * 15823 + blk[..., 1] * 9737333 + blk[..., 2] * 440817757) & 0xFFFFFFFF
    return ((loc[..., 0] + 50 * (loc[..., 1] + 50 * loc[..., 2]) + bh) & 0xFFFFFFFF) % n


def _cells(x, h):
    return torch.floor(x.to(torch.float32) / torch.tensor(h, dtype=torch.float32, device=x.device)).to(torch.int64)


def _particles(case, n, seed):
    """Positions and velocities (n, 3) on the GPU."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=torch.float32)  # noqa: E731
    sp = case["spacing"]
    ext, box, obj = _geometry(case, n)
    if case.get("blob"):
        size = torch.tensor(box, device=DEV)
        blob = torch.randn(case["blob"], 3, generator=g, device=DEV) * 0.1 + 0.5 * size
        x = torch.cat([rand(n - case["blob"], 3) * size, blob])
        x = torch.minimum(torch.maximum(x, torch.zeros_like(x)), size)
    else:
        d = [int(round(e / sp)) for e in ext]
        while True:
            k = torch.arange(d[0] * d[1] * d[2], device=DEV)
            x = torch.stack([k % d[0], (k // d[0]) % d[1], k // (d[0] * d[1])], 1).to(torch.float32)
            x = (x + 0.5 + 0.2 * (rand(len(k), 3) - 0.5)) * sp
            if obj and obj[0] == SHAPE_SPHERE:  # no fluid in the obstacle
                c = torch.tensor(obj[2], device=DEV, dtype=torch.float32)
                x = x[((x - c) ** 2).sum(1) > (obj[1][0] + 0.6 * _h(case)) ** 2]
            if len(x) >= n:
                break
            d[2] += max(1, d[2] // 8)
        x = x[:n].contiguous()
    v = torch.zeros_like(x)
    if case["speed"]:
        ph = rand(3) * 6.2831853
        k = [2 * math.pi / e for e in ext]
        v[:, 0] = torch.sin(k[1] * x[:, 1] + ph[0]) * torch.cos(k[2] * x[:, 2] + ph[1])
        v[:, 1] = torch.sin(k[2] * x[:, 2] + ph[1]) * torch.cos(k[0] * x[:, 0] + ph[2])
        v[:, 2] = torch.sin(k[0] * x[:, 0] + ph[2]) * torch.cos(k[1] * x[:, 1] + ph[0])
        v *= case["speed"]
    if case["sorted"]:  # a checkpoint of a running model is in its spatial order
        order = torch.argsort(_keys(_cells(x, _h(case)), n), stable=True)
        x, v = x[order].contiguous(), v[order].contiguous()
    return x, v


def _params(case, n, box):
    sim = SimulationParameters((0.0, 0.0, -9.81), _h(case))
    sph = SPHParameters(1.0, 1, n, case["dt"], 1000.0, box, (0.0, 0.0, 0.0))
    return sim, sph, WCSPHParameters(1e4, case.get("stiffness", 50.0), 7.0, case["viscosity"])


def _analytic(obj, res):
    return AnalyticObject(obj[0], obj[1], position=obj[2], resolution=(res,) * 3)


def _model(case, n):
    _, box, obj = _geometry(case, n)
    m = WCSPHWithBoundaryModel(*_params(case, n, box))
    if obj:
        m.add_analytic_object(_analytic(obj, case["res"]))
    if case.get("slots", 128) != 128:
        m.set_neighbor_capacity(case["slots"])
    if case.get("skin", 0.05) != 0.05:
        m.set_skin(case["skin"])
    return m


_streams = []


def _stream():
    """The program's one stream: its models run one after the other on it."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


class _DeviceArray:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n, 4), "typestr": "<f4", "data": (ptr, False), "version": 3}


def _resident(case, n, seed):
    """A model on a torch stream, its state as torch tensors, and the checkpoint it starts from."""
    x, v = _particles(case, n, seed)
    m = _model(case, n)
    stream = _stream()
    m.set_stream(stream.cuda_stream)
    ids = torch.arange(n, device=DEV, dtype=torch.int32).view(torch.float32)
    p, q = (torch.as_tensor(_DeviceArray(a, n), device=DEV) for a in m.device_state())
    return dict(m=m, stream=stream, pos=p, vel=q, pos0=torch.cat([x, ids[:, None]], 1),
                vel0=torch.cat([v, torch.zeros(n, 1, device=DEV)], 1))


def _pinned(a):
    t = torch.empty(a.shape, dtype=a.dtype, pin_memory=True)
    t.copy_(a)
    return t.numpy()


def _scenes(case, seed):
    """The batch's scenes as single cases of their own sizes."""
    rng = np.random.default_rng(3)  # the sizes are the case's, the particles the seed's
    sizes = np.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]), case["scenes"])).astype(int)
    nus = np.exp(rng.uniform(math.log(1e-3), math.log(8e-3), case["scenes"]))
    ks = rng.uniform(20.0, 100.0, case["scenes"])
    return [(dict(kind="sim", spacing=case["spacing"], ratio=case["ratio"], speed=0.0, dt=case["dt"],
                  viscosity=float(nus[s]), stiffness=float(ks[s]), object="container", res=case["res"],
                  sorted=False, substeps=case["substeps"]), int(sizes[s]), seed * 1009 + s)
            for s in range(case["scenes"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        n = case["n"]
        g = torch.Generator(device=DEV).manual_seed(seed)
        keys = torch.randint(0, n, (n,), generator=g, device=DEV, dtype=torch.int32)
        return dict(case=case, keys0=keys, pos=torch.rand(n, 3, generator=g, device=DEV),
                    vel=torch.randn(n, 3, generator=g, device=DEV), keys=torch.empty_like(keys),
                    items=torch.empty_like(keys), offsets=torch.empty_like(keys),
                    pos_out=torch.empty(n, 3, device=DEV), vel_out=torch.empty(n, 3, device=DEV))
    if kind == "batch":
        scenes = _scenes(case, seed)
        b = Batch([_params(c, n, _geometry(c, n)[1]) for c, n, _ in scenes])
        state, off = [], 0
        for s, (c, n, sd) in enumerate(scenes):
            b.add_analytic_object(s, _analytic(_geometry(c, n)[2], c["res"]))
            state.append(tuple(_pinned(a) for a in _particles(c, n, sd)) + (off,))
            off += n
        return dict(case=case, b=b, state=state, n=off)
    n = case["n"]
    if kind == "frame":
        x, v = _particles(case, n, seed)
        empty = lambda *s: torch.empty(*s, pin_memory=True).numpy()  # noqa: E731
        return dict(case=case, m=_model(case, n), pos=_pinned(x), vel=_pinned(v),
                    out={"positions": empty(n, 3), "velocities": empty(n, 3), "densities": empty(n)})
    s = dict(case=case, **_resident(case, n, seed))
    if kind == "adjoint":
        s["rollout"] = Rollout(s["m"], case["substeps"], case["every"])
        s["seed_grad"] = _loss_gradient(case, seed).cpu().numpy().astype(np.float32)
    if kind == "view":
        s["pos"].copy_(s["pos0"])
        s["vel"].copy_(s["vel0"])
        lo, hi = _view_box(case)
        mid = 0.5 * (lo + hi)
        size = float((hi - lo).max())
        s["lo"], s["hi"] = lo, hi
        s["view"] = look_at(mid + size * np.array([1.1, -1.3, 0.8]), mid)
        s["proj"] = perspective(0.8, case["width"] / case["height"], 0.01 * size, 10.0 * size)
    return s


def _view_box(case):
    ext, _, _ = _geometry(case, case["n"])
    return np.zeros(3, np.float32), np.asarray(ext, np.float32)


def _grid_res(case):
    return (2 * case["grid"], case["grid"], case["grid"])


def _loss_gradient(case, seed):
    """d loss / d final positions, by id: of a mean squared error."""
    g = torch.Generator(device=DEV).manual_seed(seed + 77)
    n = case["n"]
    return (torch.randn(n, 3, generator=g, device=DEV) * (0.01 / n)).to(torch.float32)


# ---------------------------------------------------------------- one pass


def _by_id(s):
    ids = s["pos"].view(torch.int32)[:, 3].long()
    x, v = torch.empty_like(s["pos0"]), torch.empty_like(s["vel0"])
    x[ids] = s["pos"]
    v[ids] = s["vel"]
    return {"positions": x[:, :3], "velocities": v[:, :3]}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "frame":
        out = s["m"].step_host(s["pos"], s["vel"], case["substeps"], s["out"])
        if case["substeps"] > 1:  # a viewer that follows particles over a frame's substeps
            ids = s["m"].get_ids()
            by_id = {k: np.empty_like(a) for k, a in out.items()}
            for k, a in out.items():
                by_id[k][ids] = a
            out = by_id
        return dict(out)
    if kind == "sort":
        n = case["n"]
        stream = torch.cuda.current_stream().cuda_stream
        s["keys"].copy_(s["keys0"])
        primitives.sort_pairs(s["items"].data_ptr(), s["keys"].data_ptr(), n, n - 1, stream)
        primitives.spatial_offsets(s["keys"].data_ptr(), s["offsets"].data_ptr(), n, stream)
        for a in ("pos", "vel"):
            primitives.reorder_float3(s["items"].data_ptr(), s[a].data_ptr(), s[a + "_out"].data_ptr(), n, stream)
        return {"keys": s["keys"], "order": s["items"], "offsets": s["offsets"],
                "positions": s["pos_out"], "velocities": s["vel_out"]}
    if kind == "batch":
        b = s["b"]
        for k, (x, v, _) in enumerate(s["state"]):
            b.set_particle_state(k, x, v)
        b.substeps(case["substeps"])
        got, ids = [], []
        for k, (_, _, off) in enumerate(s["state"]):
            got.append(b.copy_data_buffers(k))
            ids.append(b.get_ids(k).astype(np.int64) + off)
        ids = torch.from_numpy(np.concatenate(ids))
        out = {}
        for key in ("positions", "velocities", "densities"):
            a = torch.from_numpy(np.concatenate([d[key] for d in got]))
            out[key] = torch.empty_like(a)
            out[key][ids] = a
        return out
    if kind == "view":
        img = s["m"].render_particles(s["view"], s["proj"], case["width"], case["height"],
                                      quad_side=2.0 * case["spacing"], depth_radius=case["spacing"],
                                      v_max=max(case["speed"], 0.1))
        grid = s["m"].density_grid(s["lo"], s["hi"], _grid_res(case))
        march = render_density_raymarch(grid / np.float32(1000.0), 0.5 * (s["lo"] + s["hi"]),
                                        0.5 * (s["hi"] - s["lo"]), s["view"], s["proj"],
                                        case["width"], case["height"],
                                        step=float((s["hi"] - s["lo"]).max()) / 100.0, emission=2.0)
        return {"image": img, "grid": grid, "march": march}
    with torch.cuda.stream(s["stream"]):
        s["pos"].copy_(s["pos0"])
        s["vel"].copy_(s["vel0"])
        if kind == "sim":
            s["m"].substeps(case["substeps"])
            return _by_id(s)
        s["rollout"].forward()
        g = s["rollout"].backward(s["seed_grad"])
        return {"final": s["rollout"].final_positions_by_id(), **g}


# ---------------------------------------------------------------- what a pass cannot do without


def _step_work(n, ratio, substeps):
    """The state in (24 B a particle) and out (24 B) each substep; per neighbour within h about 15
    operations for the density and 40 for the forces."""
    near = 4.0 / 3.0 * math.pi / ratio ** 3
    return {"bytes": 48.0 * n * substeps, "flops": 55.0 * near * n * substeps}


def work(case):
    kind = case["kind"]
    if kind == "sort":
        return {"bytes": (4 + 4 + 4 + 4 + 48) * float(case["n"]), "flops": 0.0}
    if kind == "view":
        px, nodes = case["width"] * case["height"], 2 * case["grid"] ** 3
        return {"bytes": 24.0 * case["n"] + 20.0 * px + 8.0 * nodes, "flops": 0.0}
    if kind == "batch":
        return _step_work(sum(n for _, n, _ in _scenes(case, 0)), case["ratio"], case["substeps"])
    w = _step_work(case["n"], case["ratio"], case["substeps"])
    if kind == "frame":
        w["bytes"] += 4.0 * case["n"]  # the densities
    if kind == "adjoint":
        w = {"bytes": 2.0 * w["bytes"], "flops": 4.0 * w["flops"]}
    if case.get("blob"):  # the blob's pairs: n^2 times the overlap of the Gaussian with itself
        w["flops"] += 55.0 * case["substeps"] * case["blob"] ** 2 * 4.0 / 3.0 * math.pi * _h(case) ** 3 / (
            8.0 * math.pi ** 1.5 * 0.1 ** 3)
    return w


# ---------------------------------------------------------------- the same in 64 bits


def _grids(obj, res, h):
    """The SDF and volume map of an analytic object at its grid's nodes, as the generator defines
    them: 0.8 x the 16-point Gauss-Legendre integral of gamma over the ball of radius h."""
    shape, size, _ = obj
    e = [size[0]] * 3 if shape == SHAPE_SPHERE else list(size)
    margin = _f32(8.0 * h)
    lo = [_f32(_f32(-a) - margin) for a in e]
    side = [_f32(_f32(_f32(a) - _f32(-a)) + _f32(2.0 * margin)) for a in e]
    step = [_f32(_f32(_f32(l + s) - l) / _f32(res - 1)) for l, s in zip(lo, side)]
    k = torch.arange(res, device=DEV, dtype=F64)
    ax = [(k * st + l).to(torch.float32) for st, l in zip(step, lo)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    nodes = torch.stack([x, y, z], -1).reshape(-1, 3)

    def sdf(p):
        p = p.to(F64)
        if shape == SHAPE_SPHERE:
            return torch.sqrt((p * p).sum(-1)) - size[0]
        q = p.abs() - torch.tensor(size, device=DEV, dtype=F64)
        box = torch.sqrt((q.clamp_min(0) ** 2).sum(-1)) + q.amax(-1).clamp_max(0)
        return box if shape != SHAPE_CONTAINER else -box

    d = sdf(nodes)
    t, w = np.polynomial.legendre.leggauss(16)
    tq = torch.tensor(t * h, device=DEV, dtype=torch.float32)
    wq = torch.tensor(w * h, device=DEV, dtype=F64)
    off = torch.stack(torch.meshgrid(tq, tq, tq, indexing="ij"), -1).reshape(-1, 3)
    wt = (wq[:, None, None] * wq[None, :, None] * wq[None, None, :]).reshape(-1)
    keep = (off.to(torch.float32) ** 2).sum(1) <= torch.tensor(h, dtype=torch.float32, device=DEV) ** 2
    off, wt = off[keep], wt[keep]
    vm = torch.where(d < 0, wt.sum(), torch.zeros_like(d))
    near = torch.nonzero((d >= -1.01 * h - 1e-5) & (d <= 2.0 * h)).reshape(-1)
    for c in near.split(16384):
        q = sdf(nodes[c][:, None, :] + off[None]) / h
        gam = torch.where(q <= 0, torch.ones_like(q), torch.where(
            q <= 0.5, 6 * q ** 3 - 6 * q ** 2 + 1, 2 * (1 - q).clamp_min(0) ** 3))
        vm[c] = gam @ wt
    f = lambda a: a.to(torch.float32).to(F64)  # noqa: E731
    return dict(pos=obj[2], lo=torch.tensor(lo, device=DEV, dtype=F64), side=torch.tensor(side, device=DEV, dtype=F64),
                res=res, sdf=f(d), vm=f(0.8 * vm))


def _sample(grid, o, l):
    val, n = 0.0, o["res"]
    x = (n - 1.0) * (l - o["lo"]) / o["side"]
    f = torch.floor(x.detach()).clamp(0, n - 2)
    t, c = x - f, f.long()
    for b in range(8):
        d = [(b >> a) & 1 for a in range(3)]
        wgt = 1.0
        for a in range(3):
            wgt = wgt * (t[:, a] if d[a] else 1.0 - t[:, a])
        val = val + grid[(c[:, 0] + d[0]) + n * ((c[:, 1] + d[1]) + n * (c[:, 2] + d[2]))] * wgt
    return val


def _constants(case, n):
    h = _h(case)
    _, box, obj = _geometry(case, n)
    return dict(h=h, n=n, cubic=8.0 / (math.pi * h ** 3), grad=48.0 / (math.pi * h ** 5), mass=100.0 * h ** 3,
                rho0=1000.0, wall=1e4, dt=_f32(case["dt"]), g=torch.tensor([0.0, 0.0, _f32(-9.81)], device=DEV, dtype=F64),
                lo=torch.zeros(3, device=DEV, dtype=F64), hi=torch.tensor([_f32(b) for b in box], device=DEV, dtype=F64),
                nu=torch.tensor(_f32(case["viscosity"]), device=DEV, dtype=F64),
                k=torch.tensor(_f32(case.get("stiffness", 50.0)), device=DEV, dtype=F64),
                obj=_grids(obj, case["res"], h) if obj else None)


def _W(r, P):
    q = r / P["h"]
    return P["cubic"] * torch.where(q > 0.5, 2.0 * (1.0 - q).clamp_min(0) ** 3, 6.0 * q ** 3 - 6.0 * q ** 2 + 1.0)


def _dW(r, P):
    q = r / P["h"]
    return P["grad"] * torch.where(q > 0.5, -((1.0 - q).clamp_min(0) ** 2), q * (3.0 * q - 2.0))


def _boundary(x, P):
    o, h = P["obj"], P["h"]
    psi, G = torch.zeros_like(x[:, 0]), torch.zeros_like(x)
    if o is None:
        return psi, G
    l = x - torch.tensor([_f32(a) for a in o["pos"]], device=DEV, dtype=F64)
    inside = ((l >= o["lo"]) & (l <= o["lo"] + o["side"])).all(1)
    with torch.no_grad():
        dist = _sample(o["sdf"], o, l)
        act = torch.nonzero(inside & (dist >= 0) & (dist < h) & (_sample(o["vm"], o, l) > 0)).reshape(-1)
    if not len(act):
        return psi, G
    l = l[act]
    e = 0.1 * h * torch.eye(3, device=DEV, dtype=F64)
    g = torch.stack([(_sample(o["sdf"], o, l + e[a]) - _sample(o["sdf"], o, l - e[a])) / (0.2 * h)
                     for a in range(3)], 1)
    nrm = g / torch.sqrt((g * g).sum(1, keepdim=True))
    d = (_sample(o["sdf"], o, l) + 0.125 * h).clamp_min(0.5 * h)
    vol = _sample(o["vm"], o, l)
    return psi.index_add(0, act, vol * _W(d, P)), G.index_add(0, act, (vol * _dW(d, P))[:, None] * nrm)


def _pairs(x, P):
    """Chunks of the ordered pairs (i, j), i != j, within h, as often as the 27-cell walk of the
    spatial hash meets them; and how often it meets each particle itself."""
    n, h = P["n"], P["h"]
    cells = _cells(x, h)
    keys = _keys(cells, n)
    order = torch.argsort(keys, stable=True)
    sk = keys[order]
    off = torch.stack(torch.meshgrid(*[torch.arange(-1, 2, device=DEV)] * 3, indexing="ij"), -1).reshape(-1, 3)
    me = torch.zeros(n, device=DEV, dtype=F64)
    out = []
    for a in range(0, n, 65536):
        nk = _keys(cells[a:a + 65536, None, :] + off[None], n)
        me[a:a + 65536] = (nk == keys[a:a + 65536, None]).sum(1).to(F64)
        b = torch.searchsorted(sk, nk.reshape(-1))
        cnt = torch.searchsorted(sk, nk.reshape(-1), right=True) - b
        rows = torch.repeat_interleave(torch.arange(len(cnt), device=DEV), cnt)
        j = order[b[rows] + torch.arange(len(rows), device=DEV) - (torch.cumsum(cnt, 0) - cnt)[rows]]
        i = rows // 27 + a
        r2 = ((x[i] - x[j]) ** 2).sum(1)
        keep = (r2 <= h * h) & (i != j)
        out.append((i[keep], j[keep]))
    return out, me


def _substep(x, v, P):
    """One substep; returns the new positions and velocities and the densities."""
    pairs, me = _pairs(x.detach(), P)
    psi, G = _boundary(x, P)
    rho = me * P["mass"] * P["cubic"] + P["rho0"] * psi
    for i, j in pairs:
        d = x[i] - x[j]
        rho = rho.index_add(0, i, P["mass"] * _W(torch.sqrt((d * d).sum(1).clamp_min(1e-300)), P))
    pr = P["k"] * ((rho.clamp_min(P["rho0"]) / P["rho0"]) ** 7 - 1.0)
    pd, mr = pr / (rho * rho), P["mass"] / rho.clamp_min(1e-6)
    acc = P["g"] - ((pd + pr / P["rho0"] ** 2) * P["rho0"])[:, None] * G
    for i, j in pairs:
        d = x[i] - x[j]
        r2 = (d * d).sum(1).clamp_min(1e-300)
        r = torch.sqrt(r2)
        u = _dW(r, P) / r
        s = -P["mass"] * (pd[i] + pd[j]) * u
        s = s + 10.0 * P["nu"] * mr[j] * ((v[i] - v[j]) * d).sum(1) * u / (r2 + 0.01 * P["h"] ** 2)
        acc = acc.index_add(0, i, torch.where(r > 1e-9, s, torch.zeros_like(s))[:, None] * d)
    acc = acc - P["wall"] * ((x - P["lo"]).clamp_max(0) - (P["hi"] - x).clamp_max(0))
    v = v + acc * P["dt"]
    return x + v * P["dt"], v, rho


def _roll(case, n, seed):
    x, v = _particles(case, n, seed)
    P = _constants(case, n)
    order = torch.argsort(_keys(_cells(x, P["h"]), n), stable=True)
    x, v = x.to(F64), v.to(F64)
    for _ in range(case["substeps"]):
        x, v, rho = _substep(x, v, P)
    return x, v, rho, order


def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":
        s = prepare(case, seed)
        keys, order = torch.sort(s["keys0"], stable=True)
        first = torch.full((case["n"],), case["n"], dtype=torch.int32, device=DEV)
        k, cnt = torch.unique_consecutive(keys, return_counts=True)
        first[k.long()] = (torch.cumsum(cnt, 0) - cnt).to(torch.int32)
        return {"keys": keys, "order": order.to(torch.int32), "offsets": first,
                "positions": s["pos"][order].to(F64), "velocities": s["vel"][order].to(F64)}
    if kind == "view":
        return {"image": None, "grid": _exact_grid(case, seed), "march": None}
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    with torch.no_grad():
        if kind == "batch":
            parts = [_roll(c, n, sd) for c, n, sd in _scenes(case, seed)]
            return {k: torch.cat([p[a] for p in parts]) for a, k in enumerate(("positions", "velocities", "densities"))}
        x, v, rho, order = _roll(case, case["n"], seed)
    if kind == "sim":
        return {"positions": x, "velocities": v}
    if case["substeps"] == 1:  # in the model's order: stable by the key at the substep's start
        x, v, rho = x[order], v[order], rho[order]
    return {"positions": x, "velocities": v, "densities": rho}


def _exact_adjoint(case, seed):
    n = case["n"]
    x0, v0 = (a.to(F64).requires_grad_() for a in _particles(case, n, seed))
    P = _constants(case, n)
    P["nu"].requires_grad_()
    P["k"].requires_grad_()
    x, v = x0, v0
    for _ in range(case["substeps"]):
        x, v, _ = _substep(x, v, P)
    g = torch.autograd.grad(x, (v0, x0, P["nu"], P["k"]), _loss_gradient(case, seed).to(F64))
    return {"final": x.detach(), "dv0": g[0], "dx0": g[1], "dnu": float(g[2]), "dk": float(g[3])}


def _exact_grid(case, seed):
    x, _ = _particles(case, case["n"], seed)
    h = _h(case)
    lo, hi = _view_box(case)
    res = _grid_res(case)
    x = x.to(F64)
    lo = torch.tensor(lo, device=DEV, dtype=F64)
    step = (torch.tensor(hi, device=DEV, dtype=F64) - lo) / (torch.tensor(res, device=DEV, dtype=F64) - 1.0)
    base = torch.floor((x - lo) / step).long()
    rad = [int(math.ceil(h / float(s))) for s in step]
    grid = torch.zeros(res[2] * res[1] * res[0], device=DEV, dtype=F64)
    sigma = 100.0 * h ** 3 * 8.0 / (math.pi * h ** 3)
    for dz in range(-rad[2], rad[2] + 2):
        for dy in range(-rad[1], rad[1] + 2):
            for dx in range(-rad[0], rad[0] + 2):
                c = base + torch.tensor([dx, dy, dz], device=DEV)
                d = lo + c * step - x
                q = torch.sqrt((d * d).sum(1)) / h
                ok = (q <= 1.0) & (c >= 0).all(1) & (c[:, 0] < res[0]) & (c[:, 1] < res[1]) & (c[:, 2] < res[2])
                w = torch.where(q <= 0.5, 6 * q ** 3 - 6 * q ** 2 + 1, 2 * (1 - q) ** 3)
                grid.index_add_(0, torch.where(ok, c[:, 0] + res[0] * (c[:, 1] + res[1] * c[:, 2]), 0),
                                torch.where(ok, sigma * w, 0.0))
    return grid.reshape(res[2], res[1], res[0])
