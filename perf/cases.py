"""The workloads this library is timed on: what its users have it do, through
its public entry points, from the smallest calls to the largest.

A case is a dict of plain values.  ``kind`` says which path it takes:

  rollout    state in (CUDA tensors), n steps, state out: the forward solver
  host       the same through pgmpm_advance_host, state in pinned host memory
  batch      many scenes of different sizes stepped by one solver
  grad       differentiable rollout (autograd.simulate) and its gradients
  pic        autograd.MPMTimestep, the reference's PIC step, with gradients
  neighbors  spatial hash grid: build and the neighbour lists of every particle
  contact    SPH-MPM contact coupling on a solver's current particles

Particles start from a state as met in mid-simulation: uniform random
positions in a body, a smooth velocity field with its gradient as the APIC
matrix, and a smoothly strained deformation gradient.  Every pass of a rollout
starts from that state, as an optimisation or a control loop does.

``exact`` restates each path in float64 with plain torch operations.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import physgrad_b200 as pg
from physgrad_b200 import autograd

DEV = "cuda:0"
PTR_HOST, PTR_DEVICE = 0, 1
STICKY, SLIP, SEPARATE = 1, 2, 3
RHO = 1000.0
G = (0.0, -9.8, 0.0)
LONGEST = 24.0  # wavelengths per unit length of the initial fields are at most this / 2 pi


# ------------------------------------------------------------------- cases
def listed():
    return [
        # a control loop's call: a small elastic body, a few substeps per call
        dict(name="cube_4k", kind="rollout", mats="fcr", n=4096, nx=32, ny=32, nz=32, steps=5, wall=STICKY, pool=0),
        # the elastic cube on 64^3 nodes: latency-bound steps, many per call
        dict(name="cube_32k", kind="rollout", mats="fcr", n=32768, nx=64, ny=64, nz=64, steps=50, wall=STICKY, pool=0),
        # elastoplastic block beside a viscous fluid, ragged grid and count
        dict(name="plastic_150k", kind="rollout", mats="plastic", n=150001, nx=93, ny=61, nz=77, steps=10,
             wall=SEPARATE, pool=0),
        # a quarter of a million particles in a 2048^3 domain: the sparse tile pool
        dict(name="sparse_262k", kind="rollout", mats="fcr", n=262144, nx=2048, ny=2048, nz=2048, steps=10,
             wall=STICKY, pool=4096),
        # the two-material drop, the largest single scene
        dict(name="drop_2m", kind="rollout", mats="drop", n=2097152, nx=128, ny=128, nz=128, steps=20, wall=SLIP,
             pool=0),
        # a host program's frame: state in and out of pinned host memory
        dict(name="host_262k", kind="host", mats="drop", n=262144, nx=64, ny=64, nz=64, steps=20, wall=SLIP, pool=0),
        # 64 scenes of 4,096 to 262,144 particles stepped together
        dict(name="batch_64", kind="batch", scenes=64, lo=4096, hi=262144, layout=0, steps=10),
        # differentiable elastic cube: forward, and gradients of a loss on the final state
        dict(name="grad_262k", kind="grad", scenes=1, lo=262144, hi=262144, layout=0, nodes=64, steps=48, every=16),
        # system identification over a batch of scenes: short differentiable rollouts
        dict(name="grad_batch", kind="grad", scenes=12, lo=4096, hi=65536, layout=3, nodes=0, steps=24, every=8),
        # the reference's PIC step as one layer of a learned model, with its backward
        dict(name="pic_100k", kind="pic", n=100003, res=64),
        # neighbour search over every particle of a cloud
        dict(name="neighbors_2m", kind="neighbors", n=2097152, cells=128, radius=1.0),
        # fluid slab in contact with the drop's particles
        dict(name="contact_1m", kind="contact", n=1048576, nodes=96, n_sph=131072, radius=2.0),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rollout", "rollout", "rollout", "host", "batch", "grad", "grad", "pic", "neighbors",
                       "contact"])
    if kind in ("rollout", "host"):
        n = _logint(rng, 2048, 2097152 if kind == "rollout" else 400000)
        mats = rng.choice(["fcr", "drop", "plastic"])
        ppc = rng.uniform(3.0, 14.0)  # particles per cell
        edge = min(150.0, max(20.0, (n / ppc) ** (1.0 / 3.0) / 0.3))
        nx, ny, nz = (max(20, int(edge * rng.uniform(0.85, 1.2))) for _ in range(3))
        pool = 0
        if kind == "rollout" and mats != "plastic" and rng.random() < 0.2:  # a large domain, sparsely filled
            nx = ny = nz = rng.randint(512, 2048)
            pool = 32768
        # at most the drop's particle steps
        steps = max(1, min(_logint(rng, 1, 64), int(2097152 * 20 / n)))
        return dict(kind=kind, mats=mats, n=n, nx=nx, ny=ny, nz=nz, steps=steps,
                    wall=rng.choice([STICKY, SLIP, SEPARATE]), pool=pool)
    if kind == "batch":
        lo = _logint(rng, 2000, 20000)
        return dict(kind=kind, scenes=rng.randint(3, 48), lo=lo, hi=lo * rng.randint(2, 12),
                    layout=rng.randrange(1 << 20), steps=rng.randint(1, 16))
    if kind == "grad":
        if rng.random() < 0.5:
            n = _logint(rng, 4000, 262144)
            return dict(kind=kind, scenes=1, lo=n, hi=n, layout=rng.randrange(1 << 20),
                        nodes=min(72, max(24, int((n / rng.uniform(4.0, 30.0)) ** (1.0 / 3.0) / 0.3))),
                        steps=rng.randint(2, 40), every=rng.randint(2, 16))
        return dict(kind=kind, scenes=rng.randint(2, 12), lo=3000, hi=_logint(rng, 6000, 65536),
                    layout=rng.randrange(1 << 20), nodes=0, steps=rng.randint(2, 24), every=rng.randint(2, 12))
    if kind == "pic":
        return dict(kind=kind, n=_logint(rng, 2000, 400000), res=rng.randint(24, 96))
    if kind == "neighbors":
        n = _logint(rng, 20000, 2000000)
        # one to four particles per cell; wider radii on the smaller clouds
        return dict(kind=kind, n=n, cells=max(8, int((n / rng.uniform(1.0, 4.0)) ** (1.0 / 3.0))),
                    radius=rng.choice([0.5, 1.0]) if n > 300000 else rng.choice([0.5, 1.0, 1.6]))
    n = _logint(rng, 30000, 1000000)
    return dict(kind=kind, n=n, nodes=max(32, int((n / rng.uniform(4.0, 12.0)) ** (1.0 / 3.0) / 0.45)),
                n_sph=_logint(rng, 2000, 120000), radius=rng.uniform(1.0, 2.0))


# ------------------------------------------------------------------ inputs
def _f32(v):
    return float(np.float32(v))


def _materials(kind):
    if kind == "fcr":
        return [pg.createElasticMaterial(RHO, 1e4, 0.3)]
    if kind == "drop":
        return [pg.createElasticMaterial(RHO, 5e4, 0.3, pg.ConstitutiveModel.NEO_HOOKEAN),
                pg.createFluidMaterial(RHO, 0.0, 1e4)]
    return [pg.MaterialParameters(RHO, 5e4, 0.3, pg.MaterialType.ELASTOPLASTIC, pg.ConstitutiveModel.NEO_HOOKEAN,
                                  yield_stress=1.5e3),
            pg.createFluidMaterial(RHO, 2.0, 1e4)]


def _scene_state(gen, boxes, dx, amp=0.02, speed=0.5):
    """Particles in ``boxes`` [(count, lo, hi, material, fluid)] with smooth random
    velocity and displacement fields; float32 CUDA tensors."""
    xs, mats, fluid = [], [], []
    for cnt, lo, hi, mat, is_fluid in boxes:
        lo, hi = (torch.tensor(a, dtype=torch.float32, device=DEV) for a in (lo, hi))
        xs.append(lo + (hi - lo) * torch.rand(cnt, 3, generator=gen, device=DEV))
        mats.append(torch.full((cnt,), mat, dtype=torch.int32, device=DEV))
        fluid.append(torch.full((cnt,), is_fluid, dtype=torch.bool, device=DEV))
    x, mat, fluid = torch.cat(xs), torch.cat(mats), torch.cat(fluid)
    n = x.shape[0]
    eye = torch.eye(3, device=DEV)

    def field(a):
        # a sum of three plane waves per component, and its gradient
        f, grad = torch.zeros(n, 3, device=DEV), torch.zeros(n, 3, 3, device=DEV)
        for _ in range(3):
            k = (torch.rand(3, 3, generator=gen, device=DEV) - 0.5) * LONGEST
            ph = torch.rand(3, generator=gen, device=DEV) * 6.2831853
            arg = x @ k.T + ph
            f += a * torch.sin(arg)
            grad += a * torch.cos(arg)[:, :, None] * k[None]
        return f, grad

    v, gradv = field(speed / 3)
    _, gradu = field(amp / 12)
    F = eye + gradu
    J = torch.linalg.det(F.double()).clamp_min(0.1)
    F = torch.where(fluid[:, None, None], (J ** (1.0 / 3.0)).float()[:, None, None] * eye, F)
    V0 = torch.full((n,), (dx / 2) ** 3, dtype=torch.float32, device=DEV)
    return dict(x=x, v=v, C=gradv.contiguous(), F=F.contiguous(), m=RHO * V0, V0=V0, mat=mat)


def _rollout_layout(case):
    """Scene and particle boxes of a rollout case."""
    n = case["n"]
    dims = (case["nx"], case["ny"], case["nz"])
    if case["pool"]:
        # a body of ~6 particles per cell somewhere inside a large sparse domain
        dx = 1.0 / 64
        side = (n / 6.0) ** (1.0 / 3.0) * dx
        origin = tuple(-0.5 * (d // 2) * dx for d in dims)
        lo, ext = (0.05, 0.05, 0.05), (side * 3,) * 3
        rel = [((0.0, 0.0, 0.0), (1 / 3, 1 / 3, 1 / 3)), ((0.36, 0.02, 0.0), (0.66, 0.35, 1 / 3))]
    else:
        dx = 1.0 / max(dims)
        origin = (0.0, 0.0, 0.0)
        lo, ext = (0.0, 0.0, 0.0), tuple((d - 1) * dx for d in dims)
        rel = [((0.2, 0.2, 0.2), (0.5, 0.5, 0.5)), ((0.55, 0.08, 0.2), (0.85, 0.6, 0.8))]
    dt = 1e-4 if dx > 0.012 else 5e-5
    box = lambda r: ([lo[a] + r[0][a] * ext[a] for a in range(3)], [lo[a] + r[1][a] * ext[a] for a in range(3)])
    if case["mats"] == "fcr":
        one = ((0.0, 0.0, 0.0), (1 / 3, 1 / 3, 1 / 3)) if case["pool"] else ((0.3, 0.3, 0.3), (0.6, 0.6, 0.6))
        boxes = [(n, *box(one), 0, False)]
    else:
        boxes = [(n // 2, *box(rel[0]), 0, False), (n - n // 2, *box(rel[1]), 1, True)]
    return pg.Scene(dims, dx, dt, G, origin, 0, case["wall"], 3), boxes


def _batch_layout(case):
    """Scenes, counts and materials of a batch or grad case, fixed by ``layout``."""
    rng = np.random.default_rng(case["layout"])
    s = case["scenes"]
    counts = np.floor(np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"] + 0.5), s))).astype(int)
    E = rng.uniform(5e3, 5e4, s) if s > 1 else np.array([1e4])
    scenes, mats = [], []
    for c, e in zip(counts, E):
        nodes = case.get("nodes") or (32 if c < 16384 else (64 if c < 131072 else 128))
        scenes.append(pg.Scene((nodes,) * 3, 1.0 / nodes, 1e-4 if nodes <= 64 else 5e-5, G, (0.0, 0.0, 0.0), 0,
                               STICKY, 3))
        mats.append(pg.createElasticMaterial(RHO, float(e), 0.3))
    return scenes, [int(c) for c in counts], mats


def _batch_state(gen, scenes, counts):
    parts = [_scene_state(gen, [(c, (0.3,) * 3, (0.6,) * 3, i, False)], s.dx)
             for i, (s, c) in enumerate(zip(scenes, counts))]
    return {k: torch.cat([p[k] for p in parts]) for k in parts[0]}


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)
    return g


def _inputs(case, seed):
    """The tensors a pass is given, float32 on the GPU, from the seed alone."""
    gen = _gen(seed)
    kind = case["kind"]
    if kind in ("rollout", "host"):
        scene, boxes = _rollout_layout(case)
        return dict(scenes=[scene], counts=[case["n"]], mats=_materials(case["mats"]),
                    st=_scene_state(gen, boxes, scene.dx))
    if kind in ("batch", "grad"):
        scenes, counts, mats = _batch_layout(case)
        d = dict(scenes=scenes, counts=counts, mats=mats, st=_batch_state(gen, scenes, counts))
        if kind == "grad":
            n = sum(counts)
            d["target"] = d["st"]["x"] + 0.01 * torch.randn(n, 3, generator=gen, device=DEV)
        return d
    if kind == "pic":
        n, res = case["n"], case["res"]
        x = 0.2 + 0.6 * torch.rand(n, 3, generator=gen, device=DEV)
        return dict(x=x, v=torch.randn(n, 3, generator=gen, device=DEV),
                    m=0.5 + torch.rand(n, generator=gen, device=DEV),
                    g=torch.tensor(G, device=DEV) + 0.1 * torch.randn(3, generator=gen, device=DEV),
                    gx=torch.randn(n, 3, generator=gen, device=DEV), gv=torch.randn(n, 3, generator=gen, device=DEV))
    if kind == "neighbors":
        return dict(x=torch.rand(case["n"], 3, generator=gen, device=DEV))
    nodes, n = case["nodes"], case["n"]
    dx = 1.0 / nodes
    scene = pg.Scene((nodes,) * 3, dx, 5e-5, G, (0.0, 0.0, 0.0), 0, SLIP, 3)
    st = _scene_state(gen, [(n, (0.2, 0.2, 0.2), (0.65, 0.65, 0.65), 0, False)], dx)
    # a slab of SPH particles across the body's top face
    sx = torch.tensor((0.2, 0.62, 0.2), device=DEV) + torch.tensor((0.45, 0.06, 0.45), device=DEV) * torch.rand(
        case["n_sph"], 3, generator=gen, device=DEV)
    sv = 0.05 * torch.randn(case["n_sph"], 3, generator=gen, device=DEV)
    return dict(scenes=[scene], counts=[n], mats=_materials("fcr"), st=st, sx=sx, sv=sv, radius=case["radius"] * dx)


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    d["kind"] = kind
    if kind in ("rollout", "host", "batch", "grad", "contact"):
        n = sum(d["counts"])
        pool = case.get("pool") or None
        sim = d["sim"] = pg.Simulator(d["scenes"], d["counts"], d["mats"], sparse_tiles=pool)
        st = d["st"]
        d["mat"] = st["mat"] if len(d["mats"]) > 1 else None
        d["steps"] = case.get("steps")
        d["out"] = {"x": torch.empty(n, 3, device=DEV), "v": torch.empty(n, 3, device=DEV),
                    "C": torch.empty(n, 3, 3, device=DEV), "F": torch.empty(n, 3, 3, device=DEV)}
        if kind == "host":
            d["host_in"] = {k: (st[k].cpu().pin_memory() if k != "mat" or d["mat"] is not None else None) for k in st}
            d["host_out"] = {k: torch.empty_like(d["out"][k], device="cpu").pin_memory() for k in d["out"]}
            d["ptrs"] = [None if d["host_in"][k] is None else d["host_in"][k].data_ptr()
                         for k in ("x", "v", "C", "F", "m", "V0", "mat")]
            d["ptrs_out"] = [d["host_out"][k].data_ptr() for k in ("x", "v", "C", "F")]
        elif kind == "grad":
            d["every"] = case["every"]
            d["E"] = torch.tensor([m.youngs_modulus for m in d["mats"]], dtype=torch.float32, device=DEV,
                                  requires_grad=True)
            d["leaves"] = {k: st[k].clone().requires_grad_(True) for k in ("x", "v", "C", "F")}
        elif kind == "contact":
            sim.upload(st["x"], st["v"], st["C"], st["F"], st["m"], st["V0"], d["mat"])
    elif kind == "pic":
        d["res"] = case["res"]
        for k in ("x", "v", "m", "g"):
            d[k].requires_grad_(True)
    elif kind == "neighbors":
        d["grid"] = _HashGrid(1.0 / case["cells"], case["n"])
        d["radius"] = _f32(case["radius"] / case["cells"])
        d["offsets"] = torch.zeros(case["n"] + 1, dtype=torch.int64, device=DEV)
        d["indices"] = torch.zeros(int(1.1 * _list_entries(case)) + 4096, dtype=torch.int32, device=DEV)
    return d


class _HashGrid:
    """A hash grid over the unit cube through the C-ABI, on device arrays."""

    def __init__(self, cell, capacity):
        self.h = ctypes.c_void_p()
        lo, hi = (ctypes.c_float * 3)(0.0, 0.0, 0.0), (ctypes.c_float * 3)(1.0, 1.0, 1.0)
        _check(pg.lib().pgmpm_hashgrid_create(float(cell), lo, hi, int(capacity), 0, ctypes.byref(self.h)))

    def __del__(self):
        pg.lib().pgmpm_hashgrid_destroy(self.h)


def _list_entries(case):
    """Expected length of all neighbour lists together: a list holds every particle
    of the buckets its cells hash to (Morton code modulo the number of cells)."""
    c, n = case["cells"], case["n"]
    code = torch.zeros(1, dtype=torch.int64)
    for a in range(3):
        v = torch.arange(c, dtype=torch.int64)
        for mul, mask in ((0x10001, 0xFF0000FF), (0x101, 0x0F00F00F), (0x11, 0xC30C30C3), (0x5, 0x49249249)):
            v = (v * mul) & mask
        code = (code[:, None] | (v << a)[None]).reshape(-1)
    share = torch.bincount(code % c ** 3, minlength=c ** 3).double()
    return n * ((2 * math.ceil(case["radius"]) + 1) ** 3 * n / c ** 3 * float((share ** 2).mean()) + 1)


def _check(rc):
    if rc:
        raise RuntimeError(pg.lib().pgmpm_last_error().decode())


def _stream():
    return torch.cuda.current_stream().cuda_stream


# -------------------------------------------------------------------- pass
def run(d):
    kind = d["kind"]
    if kind in ("rollout", "batch"):
        st, sim, stream = d["st"], d["sim"], torch.cuda.current_stream()
        sim.upload(st["x"], st["v"], st["C"], st["F"], st["m"], st["V0"], d["mat"], stream=stream)
        sim.step(d["steps"], stream=stream)
        return dict(sim.download(d["out"], stream=stream))
    if kind == "host":
        _check(pg.lib().pgmpm_advance_host(d["sim"].handle, *d["ptrs"], d["steps"], *d["ptrs_out"],
                                           ctypes.c_void_p(_stream())))
        return d["host_out"]
    if kind == "grad":
        lv, st = d["leaves"], d["st"]
        x, v, C, F = autograd.simulate(d["sim"], lv["x"], lv["v"], d["E"], st["m"], st["V0"], d["steps"], d["every"],
                                       C0=lv["C"], F0=lv["F"], mat=d["mat"])
        loss = _loss(x, v, F, d["target"])
        g = torch.autograd.grad(loss, [lv["x"], lv["v"], lv["C"], lv["F"], d["E"]])
        return {"x": x.detach(), "v": v.detach(), "C": C.detach(), "F": F.detach(), "gx": g[0], "gv": g[1],
                "gC": g[2], "gF": g[3], "gE": g[4]}
    if kind == "pic":
        x, v = autograd.MPMTimestep.apply(d["x"], d["v"], d["m"], d["g"], d["res"], 1e-3)
        g = torch.autograd.grad([x, v], [d["x"], d["v"], d["m"], d["g"]], [d["gx"], d["gv"]])
        return {"x": x.detach(), "v": v.detach(), "gx": g[0], "gv": g[1], "gm": g[2], "gg": g[3]}
    if kind == "neighbors":
        L, h, st, x = pg.lib(), d["grid"].h, ctypes.c_void_p(_stream()), d["x"]
        n = x.shape[0]
        total = ctypes.c_int64()
        _check(L.pgmpm_hashgrid_build(h, x.data_ptr(), n, PTR_DEVICE, st))
        _check(L.pgmpm_hashgrid_neighbors(h, x.data_ptr(), n, d["radius"], d["offsets"].data_ptr(),
                                          d["indices"].data_ptr(), d["indices"].numel(), ctypes.byref(total),
                                          PTR_DEVICE, st))
        if total.value > d["indices"].numel():  # as a user's program: grow the buffer and ask again
            d["indices"] = torch.zeros(total.value, dtype=torch.int32, device=DEV)
            _check(L.pgmpm_hashgrid_neighbors(h, x.data_ptr(), n, d["radius"], d["offsets"].data_ptr(),
                                              d["indices"].data_ptr(), d["indices"].numel(), ctypes.byref(total),
                                              PTR_DEVICE, st))
        return {"offsets": d["offsets"], "indices": d["indices"]}  # the buffer's tail stays zero
    f, mf, pairs, energy = d["sim"].sph_coupling(d["sx"], d["sv"], radius=d["radius"],
                                                 stream=torch.cuda.current_stream())
    return {"sph_force": f, "mpm_force": mf, "pairs": pairs, "energy": energy}


def _loss(x, v, F, target):
    n = x.shape[0]
    return ((x - target) ** 2).sum() * (0.5 / n) + (v ** 2).sum() * (0.05 / n) + (F ** 2).sum() * (0.01 / n)


def work(case):
    kind = case["kind"]
    if kind in ("rollout", "host", "batch", "grad"):
        n = case["n"] if "n" in case else sum(_batch_layout(case)[1])
        ps = n * case["steps"]
        # a particle step: x, v, C, F (96 B) in and out, mass and volume; the
        # 27-node scatter and gather with the stress, about 1000 operations
        b, f = 200.0 * ps, 1000.0 * ps
        if kind == "grad":  # and the step's reverse: the state again, the adjoint in and out
            b, f = b + 300.0 * ps, f + 2500.0 * ps
        return {"bytes": b, "flops": f}
    if kind == "pic":
        n, nodes = case["n"], (0.6 * case["res"] + 2) ** 3
        return {"bytes": 148.0 * n + 64.0 * nodes, "flops": 27.0 * 70 * n}
    if kind == "neighbors":
        n, w = case["n"], 2 * math.ceil(case["radius"]) + 1
        return {"bytes": n * (24.0 + 16.0 + 8.0) + 4.0 * _list_entries(case), "flops": 20.0 * n * w ** 3}
    vol = 0.45 ** 3 * case["nodes"] ** 3
    pairs = 0.5 * case["n_sph"] * (case["n"] / vol) * 4.19 * case["radius"] ** 3
    return {"bytes": 44.0 * case["n"] + 36.0 * case["n_sph"], "flops": 60.0 * pairs}


# ------------------------------------------------- the same in 64-bit torch
def exact(case, seed):
    kind = case["kind"]
    if kind == "neighbors":
        return None  # whole numbers
    d = _inputs(case, seed)
    if kind == "pic":
        return _exact_pic(case, d)
    if kind == "contact":
        return _exact_contact(d)
    ranges, b = [], 0
    for c in d["counts"]:
        ranges.append((b, b + c))
        b += c
    out = {k: [] for k in ("x", "v", "C", "F")}
    grads = {k: [] for k in ("gx", "gv", "gC", "gF")}
    gE = torch.zeros(len(d["mats"]), dtype=torch.float64, device=DEV)
    n = b
    for scene, (lo, hi) in zip(d["scenes"], ranges):
        st = {k: d["st"][k][lo:hi] for k in d["st"]}
        S = _Scene64(scene, d["mats"], st, case.get("pool"))
        z = tuple(st[k].double() for k in ("x", "v", "C", "F"))
        E = torch.tensor([_f32(m.youngs_modulus) for m in d["mats"]], dtype=torch.float64, device=DEV)
        if kind != "grad":
            for _ in range(case["steps"]):
                z = S.step(*z, E)
        else:
            states = []
            for _ in range(case["steps"]):
                states.append(z)
                with torch.no_grad():
                    z = S.step(*z, E)
            t = d["target"][lo:hi].double()
            adj = [(z[0] - t) / n, z[1] * (0.1 / n), torch.zeros_like(z[2]), z[3] * (0.02 / n)]
            for s in reversed(states):
                leaves = [a.clone().requires_grad_(True) for a in s] + [E.clone().requires_grad_(True)]
                g = torch.autograd.grad(S.step(*leaves), leaves, adj)
                adj = list(g[:4])
                gE += g[4]
            for k, a in zip(grads, adj):
                grads[k].append(a)
        for k, a in zip(out, z):
            out[k].append(a)
    res = {k: torch.cat(v) for k, v in out.items()}
    if kind == "grad":
        res.update({k: torch.cat(v) for k, v in grads.items()}, gE=gE)
    return res


class _Scene64:
    """One MLS-MPM scene: P2G, grid update with walls, G2P, in float64."""

    def __init__(self, scene, mats, st, pool):
        self.n = tuple(int(a) for a in scene.n)
        self.dx, self.dt = _f32(scene.dx), _f32(scene.dt)
        t = lambda v: torch.tensor([_f32(a) for a in v], dtype=torch.float64, device=DEV)
        self.origin, self.g = t(scene.origin), t(scene.gravity)
        self.wall, self.thick = scene.boundary, scene.boundary_thickness
        self.m, self.V0 = st["m"].double(), st["V0"].double()
        self.mats, self.mat = mats, st["mat"].long()
        # the window of nodes the particles can reach (the whole grid when it is small)
        if pool:
            s = torch.floor((st["x"].double() - self.origin) / self.dx).long()
            self.w0 = [max(0, int(s[:, a].min()) - 8) for a in range(3)]
            self.wn = [min(self.n[a], int(s[:, a].max()) + 10) - self.w0[a] for a in range(3)]
        else:
            self.w0, self.wn = [0, 0, 0], list(self.n)
        self.hi = torch.tensor([k - 3 for k in self.n], device=DEV, dtype=torch.float64)
        if len(mats) == 1:
            self.mat = torch.zeros_like(self.mat)
        self.present = sorted(set(self.mat.unique().tolist()))

    def tau(self, F, C, E):
        out = torch.zeros_like(F)
        eye = torch.eye(3, dtype=F.dtype, device=F.device)
        for i in self.present:
            mt, sel = self.mats[i], self.mat == i
            every = len(self.present) == 1
            f, c = (F, C) if every else (F[sel], C[sel])
            J = _det(f)[:, None, None]
            nu = _f32(mt.poisson_ratio)
            mu, lam = E[i] / (2 * (1 + nu)), E[i] * nu / ((1 + nu) * (1 - 2 * nu))
            if mt.type == pg.MaterialType.FLUID:
                t = E[i] * J * (J - 1) * eye + J * _f32(mt.viscosity) * (c + c.transpose(1, 2))
            elif mt.type == pg.MaterialType.ELASTOPLASTIC:
                t = mu * (f @ f.transpose(1, 2) - eye) + lam * torch.log(J) * eye
                p = (t.diagonal(dim1=1, dim2=2).sum(1) / 3)[:, None, None] * eye
                vm = torch.sqrt(1.5 * ((t - p) ** 2).sum((1, 2)))[:, None, None]
                cap = J * _f32(mt.yield_stress)
                t = torch.where(vm > cap, p + cap / vm * (t - p), t)
            elif mt.model == pg.ConstitutiveModel.NEO_HOOKEAN:
                t = mu * (f @ f.transpose(1, 2) - eye) + lam * torch.log(J) * eye
            else:
                t = 2 * mu * (f - _polar(f)) @ f.transpose(1, 2) + lam * (J - 1) * J * eye
            if every:
                return t
            out = out.index_put((sel.nonzero()[:, 0],), t)
        return out

    def step(self, x, v, C, F, E):
        dx, dt = self.dx, self.dt
        D = 4.0 / (dx * dx)
        u = (x - self.origin) / dx
        s = torch.minimum(torch.floor(u.detach() - 0.5).clamp_min(0.0), self.hi)
        f = (u - s).clamp(0.5, 1.5)
        w = torch.stack([0.5 * (1.5 - f) ** 2, 0.75 - (f - 1.0) ** 2, 0.5 * (f - 0.5) ** 2])
        A = (-dt * D) * self.V0[:, None, None] * self.tau(F, C, E) + self.m[:, None, None] * C
        b = self.m[:, None] * v
        s = s.long() - torch.tensor(self.w0, device=s.device)
        wn = self.wn
        nodes = wn[0] * wn[1] * wn[2]
        grid = torch.zeros(nodes, 4, dtype=x.dtype, device=x.device)
        offs = [(i, j, k) for k in range(3) for j in range(3) for i in range(3)]
        base = (s[:, 2] * wn[1] + s[:, 1]) * wn[0] + s[:, 0]
        for i, j, k in offs:
            wt = w[i, :, 0] * w[j, :, 1] * w[k, :, 2]
            d = (torch.tensor((i, j, k), dtype=x.dtype, device=x.device) - f) * dx
            val = torch.cat([self.m[:, None], b + (A @ d[:, :, None])[:, :, 0]], 1) * wt[:, None]
            grid = grid.index_add(0, base + ((k * wn[1] + j) * wn[0] + i), val)
        m = grid[:, :1]
        gv = torch.where(m > 0, grid[:, 1:] / torch.where(m > 0, m, torch.ones_like(m)) + dt * self.g,
                         torch.zeros_like(grid[:, 1:]))
        gv = self.walls(gv)
        nv, B = torch.zeros_like(v), torch.zeros_like(C)
        for i, j, k in offs:
            wt = w[i, :, 0] * w[j, :, 1] * w[k, :, 2]
            d = (torch.tensor((i, j, k), dtype=x.dtype, device=x.device) - f) * dx
            wv = wt[:, None] * gv[base + ((k * wn[1] + j) * wn[0] + i)]
            nv = nv + wv
            B = B + wv[:, :, None] * d[:, None, :]
        nC = D * B
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        nF = (eye + dt * nC) @ F
        fluid = [i for i in self.present if self.mats[i].type == pg.MaterialType.FLUID]
        if fluid:
            J = _det(nF)
            iso = (torch.sign(J) * J.abs() ** (1.0 / 3.0))[:, None, None] * eye
            nF = torch.where((self.mat == fluid[0])[:, None, None], iso, nF)
        return x + dt * nv, nv, nC, nF

    def walls(self, gv):
        if not self.wall:
            return gv
        wn, w0, n = self.wn, self.w0, self.n
        idx = [torch.arange(wn[a], device=gv.device) + w0[a] for a in range(3)]
        shape = lambda a, t: t.reshape([wn[2] if a == 2 else 1, wn[1] if a == 1 else 1, wn[0] if a == 0 else 1])
        low = [shape(a, idx[a] < self.thick).expand(wn[2], wn[1], wn[0]).reshape(-1) for a in range(3)]
        high = [shape(a, idx[a] >= n[a] - self.thick).expand(wn[2], wn[1], wn[0]).reshape(-1) for a in range(3)]
        if self.wall == STICKY:
            anyw = low[0] | high[0] | low[1] | high[1] | low[2] | high[2]
            return torch.where(anyw[:, None], torch.zeros_like(gv), gv)
        cols = []
        for a in range(3):
            c = gv[:, a]
            hit = (low[a] | high[a]) if self.wall == SLIP else ((low[a] & (c < 0)) | (high[a] & ~low[a] & (c > 0)))
            cols.append(torch.where(hit, torch.zeros_like(c), c))
        return torch.stack(cols, 1)


def _cof(A):
    a = A.reshape(-1, 9)
    c = [a[:, 4] * a[:, 8] - a[:, 5] * a[:, 7], a[:, 5] * a[:, 6] - a[:, 3] * a[:, 8],
         a[:, 3] * a[:, 7] - a[:, 4] * a[:, 6], a[:, 2] * a[:, 7] - a[:, 1] * a[:, 8],
         a[:, 0] * a[:, 8] - a[:, 2] * a[:, 6], a[:, 1] * a[:, 6] - a[:, 0] * a[:, 7],
         a[:, 1] * a[:, 5] - a[:, 2] * a[:, 4], a[:, 2] * a[:, 3] - a[:, 0] * a[:, 5],
         a[:, 0] * a[:, 4] - a[:, 1] * a[:, 3]]
    return torch.stack(c, 1).reshape(-1, 3, 3)


def _det(A):
    return (A[:, 0] * _cof(A)[:, 0]).sum(1)


def _polar(F):
    """Rotation of F = R S by Newton's iteration X <- (X + X^-T) / 2."""
    X = F
    for _ in range(7):
        c = _cof(X)
        X = 0.5 * (X + c / (X[:, 0] * c[:, 0]).sum(1)[:, None, None])
    return X


def _exact_pic(case, d):
    res, dt = case["res"], _f32(1e-3)
    dx32 = torch.tensor(1.0, dtype=torch.float32) / torch.tensor(float(res), dtype=torch.float32)
    dx = float(dx32)
    x, v, m, g = (d[k].detach().double().requires_grad_(True) for k in ("x", "v", "m", "g"))
    # the cell is the float32 quotient's floor: the stencil jumps there
    fl = torch.floor(d["x"].detach() / dx32.to(DEV)).double()
    f = x / dx - fl
    b = fl.long() - 1

    def quad(r):
        a = r.abs()
        return torch.where(a >= 1.5, torch.zeros_like(r), torch.where(a < 0.5, 0.75 - r * r, 0.5 * (1.5 - a) ** 2))

    w = torch.stack([quad(f - (k - 1)) for k in range(3)])
    grid = torch.zeros(res ** 3, 4, dtype=torch.float64, device=DEV)
    offs = [(i, j, k) for i in range(3) for j in range(3) for k in range(3)]
    base = (b[:, 2] * res + b[:, 1]) * res + b[:, 0]
    for i, j, k in offs:
        wm = (w[i, :, 0] * w[j, :, 1] * w[k, :, 2] * m)[:, None]
        grid = grid.index_add(0, base + ((k * res + j) * res + i), torch.cat([wm, wm * v], 1))
    gm = grid[:, :1]
    ok = gm > 1e-10
    gvel = torch.where(ok, grid[:, 1:] / torch.where(ok, gm, torch.ones_like(gm)) + dt * g,
                       torch.zeros_like(grid[:, 1:]))
    nv = torch.zeros_like(v)
    for i, j, k in offs:
        nv = nv + (w[i, :, 0] * w[j, :, 1] * w[k, :, 2])[:, None] * gvel[base + ((k * res + j) * res + i)]
    nx = x + dt * nv
    gr = torch.autograd.grad([nx, nv], [x, v, m, g], [d["gx"].double(), d["gv"].double()])
    return {"x": nx.detach(), "v": nv.detach(), "gx": gr[0], "gv": gr[1], "gm": gr[2], "gg": gr[3]}


def _exact_contact(d):
    """Contact forces of every pair closer than the radius (float32 distances
    decide which pairs those are, as the reference's do)."""
    k, c, mu, r = 1e5, 1e3, _f32(0.3), _f32(d["radius"])
    x, v, sx, sv = d["st"]["x"], d["st"]["v"], d["sx"], d["sv"]
    nc = max(1, int(1.0 / r) - 1)  # cells at least one radius wide
    cell = lambda p: (p * nc).floor().long().clamp(0, nc - 1)
    cx = cell(x)
    ids = (cx[:, 0] * nc + cx[:, 1]) * nc + cx[:, 2]
    order = torch.argsort(ids)
    starts = torch.searchsorted(ids[order], torch.arange(nc ** 3 + 1, device=DEV))
    f = torch.zeros(sx.shape[0], 3, dtype=torch.float64, device=DEV)
    mf = torch.zeros(x.shape[0], 3, dtype=torch.float64, device=DEV)
    energy = torch.zeros((), dtype=torch.float64, device=DEV)
    cs = cell(sx)
    r32 = torch.tensor(r, dtype=torch.float32, device=DEV)
    for o in [(i, j) for i in (-1, 0, 1) for j in (-1, 0, 1)]:
        a, b = cs[:, 0] + o[0], cs[:, 1] + o[1]
        ok = (a >= 0) & (a < nc) & (b >= 0) & (b < nc)
        a, b = a.clamp(0, nc - 1), b.clamp(0, nc - 1)
        row = (a * nc + b) * nc
        # the three cells along z are neighbours in the sorted order
        s0 = starts[row + (cs[:, 2] - 1).clamp(0, nc - 1)]
        s1 = starts[row + (cs[:, 2] + 1).clamp(0, nc - 1) + 1]
        cnt = torch.where(ok, s1 - s0, torch.zeros_like(s0))
        for part in torch.arange(sx.shape[0], device=DEV).split(1 << 15):
            n = cnt[part]
            q = torch.repeat_interleave(part, n)
            if q.numel() == 0:
                continue
            first = torch.cumsum(n, 0) - n
            p = order[torch.arange(q.numel(), device=DEV) - torch.repeat_interleave(first, n) + s0[q]]
            e = x[p] - sx[q]
            d32 = torch.sqrt((e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1]) + e[:, 2] * e[:, 2])
            near = d32 < r32
            q, p = q[near], p[near]
            e = x[p].double() - sx[q].double()
            dist = e.norm(dim=1)
            pen = r - dist
            energy = energy + (0.5 * k * pen * pen).sum()
            nrm = e / dist[:, None]
            dv = v[p].double() - sv[q].double()
            vn = (dv * nrm).sum(1)
            force = nrm * (k * pen + c * vn)[:, None]
            t = dv - nrm * vn[:, None]
            ts = t.norm(dim=1)
            fr = torch.where((ts > 1e-6)[:, None], t / ts.clamp_min(1e-30)[:, None] * (-mu * k * pen)[:, None],
                             torch.zeros_like(t))
            force = force + fr
            f.index_add_(0, q, -force)
            mf.index_add_(0, p, force)
    return {"sph_force": f, "mpm_force": mf, "pairs": None, "energy": float(energy)}
