"""Sizes at which the step's kernels can go wrong: the edges of their particle
and tile blocks, empty and one-tile scenes, single particles.

Tolerances are those of the batched and split-kernel tests of the same
quantities: two runs of one scene through different kernels differ by FP32
summation order only, x <= 1e-6 absolute, v <= 1e-4 * max|v|, F <= 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene_state(rng, N, n, dx, margin=1.2):
    lo, hi = margin * dx, (np.asarray(n) - 1 - margin) * dx
    V0 = np.full(N, (dx / 2) ** 3, np.float32)
    return dict(x=rng.uniform(lo, hi, (N, 3)).astype(np.float32), v=rng.normal(0, 0.5, (N, 3)).astype(np.float32),
                C=rng.normal(0, 1.0, (N, 9)).astype(np.float32),
                F=(np.eye(3).ravel() + rng.normal(0, 0.02, (N, 9))).astype(np.float32),
                m=(1000 * V0).astype(np.float32), V0=V0)


def _close(a, b):
    assert np.abs(a["x"] - b["x"]).max(initial=0.0) <= 1e-6
    assert np.abs(a["v"] - b["v"]).max(initial=0.0) <= 1e-4 * np.abs(b["v"]).max(initial=0.0) + 1e-7
    assert np.abs(a["F"] - b["F"]).max(initial=0.0) <= 1e-5


def test_many_small_scenes_find_their_particles_and_tiles(gpu):
    """Scenes that begin inside the scene table's blocks: empty ones, single
    particles, block-size counts, grids of one and of a few tiles."""
    rng = np.random.default_rng(5)
    counts = [0, 1, 127, 128, 129, 3, 0, 0, 64, 257, 2, 1, 500, 31, 0, 640, 1, 0]
    scenes, mats, sts = [], [], []
    for i, c in enumerate(counts):
        n = (4 + i % 5, 4 + (3 * i) % 9, 4 + (2 * i) % 7)
        scenes.append(gpu.Scene(n, 1.0 / 16, 1e-4, (0.0, -9.8, 0.0), (0.0, 0.0, 0.0), 0, 1, 1))
        mats.append(gpu.createElasticMaterial(1000.0, 5e3 + 500.0 * i, 0.3))
        sts.append(_scene_state(rng, c, n, 1.0 / 16))
    cat = {k: np.concatenate([s[k] for s in sts]) for k in sts[0]}
    ids = np.concatenate([np.full(c, i, np.int32) for i, c in enumerate(counts)])
    sim = gpu.Simulator(scenes, counts, mats)
    sim.upload(cat["x"], cat["v"], cat["C"], cat["F"], cat["m"], cat["V0"], ids)
    sim.step(6)
    out, b = sim.download(), 0
    for s, c, m, st in zip(scenes, counts, mats, sts):
        if c:
            one = gpu.Simulator([s], [c], [m])
            one.upload(st["x"], st["v"], st["C"], st["F"], st["m"], st["V0"])
            one.step(6)
            _close({k: v[b:b + c] for k, v in out.items()}, one.download())
        b += c


@pytest.mark.parametrize("N,n,boundary", [(1, (4, 4, 4), 0), (33, (5, 4, 7), 1), (255, (20, 11, 6), 2),
                                          (2049, (35, 35, 35), 1), (5000, (66, 34, 70), 3)])
def test_sorts_inside_a_call_equal_single_step_calls(gpu, N, n, boundary):
    """A call of several steps counts each step's keys in the G2P before it;
    calls of one step count them in the sort.  Both give the same particles,
    and a sorted order that is a permutation with sorted keys."""
    from physgrad_b200 import _capi as C
    rng = np.random.default_rng(N)
    dx = 1.0 / 32
    scene = gpu.Scene(n, dx, 1e-3, (0.3, -9.8, 0.1), (0.0, 0.0, 0.0), 0, boundary, 1)
    st = _scene_state(rng, N, n, dx)
    st["v"] *= 4.0  # a tenth of the particles change cell in a step
    mats = [gpu.createElasticMaterial(1000.0, 1e3, 0.3)]
    a, b = gpu.Simulator([scene], [N], mats), gpu.Simulator([scene], [N], mats)
    for s in (a, b):
        s.upload(st["x"], st["v"], st["C"], st["F"], st["m"], st["V0"])
    for calls in ((5, (1, 1, 1, 1, 1)), (2, (1, 1)), (1, (1,)), (3, (2, 1))):
        keys = a.get_array(C.ARRAY_KEYS)
        if calls[0] == 1:
            before = keys
        a.step(calls[0])
        for k in calls[1]:
            b.step(k)
        if calls[0] == 1:  # the sort of this step is that of the keys before it
            order, sk = a.get_array(C.ARRAY_SORTED_ORDER), a.get_array(C.ARRAY_SORTED_KEYS)
            assert np.array_equal(np.sort(order), np.arange(N)) and np.array_equal(before[order], np.sort(before))
            assert np.array_equal(sk, np.sort(before))
    assert a.status() == b.status()
    _close(a.download(), b.download())


@pytest.mark.parametrize("calls", [[1] * 7, [2] * 5, [5, 5, 3, 5, 5, 5, 3, 3, 3], [64, 64, 64, 64], [131, 146, 17, 200]])
@pytest.mark.parametrize("sparse", [False, True])
def test_steps_launched_one_by_one_and_in_graphs_agree(gpu, calls, sparse):
    """Calls of equal and of changing lengths, which run step by step, as a
    graph per step, per call or per 16 steps: against launches without graphs.
    The particles are free (no stress, no gravity), so the difference of two
    runs grows with the steps' rounding only: half an ulp of x (below 1.4) per
    step on each side, 4 ulp of the largest v.  A step more or less moves the
    fastest particles by dt |v| = 3e-4."""
    rng = np.random.default_rng(11)
    N, n = 700, (22, 21, 20)
    dx = 1.0 / 16
    scene = gpu.Scene(n, dx, 2e-4, (0.0, 0.0, 0.0), (0.0, 0.0, 0.0), 0, 0, 0)
    st = _scene_state(rng, N, n, dx, margin=4.0)
    mats = [gpu.createElasticMaterial(1000.0, 0.0, 0.3)]
    outs = []
    for graph in (1, 0):
        sim = gpu.Simulator([scene], [N], mats, sparse_tiles=2048 if sparse else None)
        sim.set_tuning(use_graph=graph)
        sim.upload(st["x"], st["v"], st["C"], st["F"], st["m"], st["V0"])
        for k in calls:
            sim.step(k)
        assert sim.status() == 0
        assert sim.metrics()["total_steps"] == sum(calls)
        outs.append(sim.download())
    ulps = sum(calls) * 2.0 ** -23
    assert np.abs(outs[0]["x"] - outs[1]["x"]).max() <= 1.4 * ulps + 1e-6
    assert np.abs(outs[0]["v"] - outs[1]["v"]).max() <= (4 * ulps + 1e-6) * np.abs(outs[1]["v"]).max()


@pytest.mark.parametrize("counts", [[1], [64], [1, 0, 3], [700], [5, 900, 2, 1, 40], [2000, 1]])
@pytest.mark.parametrize("sparse", [False, True])
def test_p2g_of_uneven_cells_equals_thread_per_cell(gpu, counts, sparse):
    """Cells of very different counts, at tile corners and on the tiles' seams:
    the grid of one step against the P2G with one thread per cell.  A node
    sums at most n = all particles' terms, so two orders of summation differ
    by at most n 2^-23 of the sum of the terms' sizes, bounded by n 2^-23
    times the largest nodal mass (and momentum, whose terms are bounded by
    m (|v| + |C| dx), 4 units of velocity here)."""
    rng = np.random.default_rng(len(counts) + sum(counts))
    n, dx = (23, 22, 21), 1.0 / 16
    xs = []
    for i, c in enumerate(counts):
        # origins on a tile's first cell, its last cell, and in between
        cell = np.array([[4, 4, 4], [7, 7, 7], [8, 7, 4], [11, 8, 8], [0, 0, 0], [19, 18, 17]])[i % 6]
        xs.append((cell + 0.5 + rng.uniform(0.05, 0.95, (c, 3))) * dx)
    x = np.concatenate(xs).astype(np.float32)
    N = len(x)
    V0 = np.full(N, (dx / 2) ** 3, np.float32)
    scene = gpu.Scene(n, dx, 1e-4, (0.0, 0.0, 0.0), (0.0, 0.0, 0.0), 0, 0, 0)
    v, Cm = rng.uniform(-1, 1, (N, 3)).astype(np.float32), rng.uniform(-5, 5, (N, 9)).astype(np.float32)
    F = np.tile(np.eye(3, dtype=np.float32).ravel(), (N, 1))
    grids = []
    for variant in (4, 2):
        sim = gpu.Simulator([scene], [N], [gpu.createElasticMaterial(1000.0, 0.0, 0.3)],
                            sparse_tiles=512 if sparse and variant == 4 else None)
        if variant != 4:
            sim.set_variants(p2g_variant=variant)
        sim.upload(x, v, Cm, F, (1000 * V0).astype(np.float32), V0)
        sim.step(1)
        m, gv = sim.grid()
        grids.append((m, gv * m[:, None]))
        assert sim.status() == 0
    bound = N * 2.0 ** -23
    assert np.abs(grids[0][0] - grids[1][0]).max() <= bound * grids[1][0].max()
    assert np.abs(grids[0][1] - grids[1][1]).max() <= 4 * bound * grids[1][0].max() + 1e-12


@pytest.mark.parametrize("counts", [[1], [64], [1, 0, 3], [700], [5, 900, 2, 1, 40], [2000, 1]])
@pytest.mark.parametrize("mats", ["elastic", "mixed"])
def test_adjoint_scatter_of_uneven_cells_equals_thread_per_cell(gpu, counts, mats):
    """The reverse step from cells of very different counts, through the
    scatter over a stored payload and the one with a thread per cell.  The
    gradients are sums over at most n particles' terms, so the two orders
    differ by a few times n 2^-23 of the largest gradient (3 stages: scatter,
    grid, gather), and 1e-5 for the arithmetic of the stress adjoint."""
    rng = np.random.default_rng(len(counts) + sum(counts))
    n, dx = (23, 22, 21), 1.0 / 16
    xs = []
    for i, c in enumerate(counts):
        cell = np.array([[4, 4, 4], [7, 7, 7], [8, 7, 4], [11, 8, 8], [0, 0, 0], [19, 18, 17]])[i % 6]
        xs.append((cell + 0.5 + rng.uniform(0.1, 0.9, (c, 3))) * dx)
    x = np.concatenate(xs).astype(np.float32)
    N = len(x)
    V0 = np.full(N, (dx / 2) ** 3, np.float32)
    scene = gpu.Scene(n, dx, 1e-4, (0.0, -9.8, 0.0), (0.0, 0.0, 0.0), 0, 0, 0)
    v, Cm = rng.uniform(-1, 1, (N, 3)).astype(np.float32), rng.uniform(-5, 5, (N, 9)).astype(np.float32)
    F = (np.eye(3).ravel() + rng.normal(0, 0.02, (N, 9))).astype(np.float32)
    ms = [gpu.createElasticMaterial(1000.0, 1e4, 0.3)]
    if mats == "mixed":
        ms.append(gpu.createFluidMaterial(1000, 5.0, 1e4))
    go = {k: rng.normal(0, 1, (N, d)).astype(np.float32) for k, d in (("x", 3), ("v", 3), ("C", 9), ("F", 9))}
    res = []
    for variant in (4, 2):
        sim = gpu.Simulator([scene], [N], ms)
        if variant != 4:
            sim.set_variants(p2g_variant=variant)
        sim.upload(x, v, Cm, F, (1000 * V0).astype(np.float32), V0, (np.arange(N) % len(ms)).astype(np.int32))
        sim.forward_checkpointed(1, 1)
        res.append(sim.backward(go))
        assert sim.status() == 0
    for key in ("x", "v", "C", "F"):
        a, b = np.asarray(res[0][key]).ravel(), np.asarray(res[1][key]).ravel()
        assert np.abs(a - b).max() <= (3 * N * 2.0 ** -23 + 1e-5) * np.abs(b).max(), key


@pytest.mark.parametrize("N", [1, 31, 32, 33, 255, 257, 1000])
@pytest.mark.parametrize("device", [False, True])
def test_upload_download_round_trip(gpu, N, device):
    """The state comes back bit for bit in upload order, whatever is left out
    on the way in (v, C zero, F identity) or asked for on the way out."""
    import torch
    rng = np.random.default_rng(N)
    dx = 1.0 / 32
    st = _scene_state(rng, N, (20, 24, 28), dx)
    scene = gpu.Scene((20, 24, 28), dx, 1e-4)
    sim = gpu.Simulator([scene], [N], [gpu.createElasticMaterial(1000.0, 1e4, 0.3)])
    up = (lambda a: None if a is None else torch.tensor(a, device="cuda")) if device else (lambda a: a)

    def down(names):
        if not device:
            return {k: a.reshape(N, -1) for k, a in sim.download().items() if k in names}
        # records that are not 16-byte aligned, and words around them that must stay
        bufs = {k: torch.full((N * w + 3,), 7.0, device="cuda") for k, w in (("x", 3), ("v", 3), ("C", 9), ("F", 9))}
        out = {k: bufs[k][1:1 + N * (3 if k in "xv" else 9)] for k in names}
        sim.download(out)
        torch.cuda.synchronize()
        for k in names:
            assert bufs[k][0] == 7.0 and torch.all(bufs[k][-2:] == 7.0)
        return {k: a.cpu().numpy().reshape(N, -1) for k, a in out.items()}

    for given in (("x", "v", "C", "F"), ("x",), ("x", "F"), ("x", "v")):
        sim.upload(*(up(st[k]) if k in given else None for k in ("x", "v", "C", "F")), up(st["m"]), up(st["V0"]))
        want = {k: st[k] if k in given else np.zeros_like(st[k]) for k in ("x", "v", "C", "F")}
        if "F" not in given:
            want["F"] = np.tile(np.eye(3, dtype=np.float32).ravel(), (N, 1))
        for names in (("x", "v", "C", "F"),) + ((("v",), ("F", "x"), ("C",)) if device else ()):
            got = down(names)
            for k in names:
                assert np.array_equal(got[k], want[k].reshape(N, -1)), (given, names, k)


@pytest.mark.parametrize("n_near", [1, 40, 193, 700])
def test_pic_step_routes_agree(gpu, n_near):
    """launch_mpm_timestep_* sort by bins from ~8 cells per particle on and by
    radix below.  The same particles (partly on and outside the grid's faces)
    with few and with many others far away take the two routes; results and
    gradients agree to FP32 rounding: 1e-6 of the largest value of a field,
    times 8 for the terms of a node's sums (<= 700 / 27 per cell on average)."""
    import torch
    from physgrad_b200 import autograd
    rng = np.random.default_rng(n_near)
    res, dx = 108, 1.0 / 108
    near = rng.uniform(0.0, 9.0, (n_near, 3)) * dx
    near[: n_near // 8 + 1] = rng.uniform(-3.0, 1.0, (n_near // 8 + 1, 3)) * dx  # outside and at the lowest nodes
    outs = []
    for n_far in (50, 40000):  # 27^3 tiles: radix up to ~26 K particles
        far = 0.4 + rng.uniform(0.0, 0.5, (n_far, 3))
        x = np.concatenate([near, far]).astype(np.float32)
        r2 = np.random.default_rng(7)
        vals = r2.normal(0, 1, (n_near, 10)).astype(np.float32)
        pad = lambda a, w: np.concatenate([a.reshape(n_near, w), np.ones((n_far, w), np.float32)])
        t = lambda a: torch.tensor(a, device="cuda")
        xs, vs = t(x).requires_grad_(True), t(pad(vals[:, :3], 3)).requires_grad_(True)
        m = t(pad(0.5 + np.abs(vals[:, 3]), 1)[:, 0].copy()).requires_grad_(True)
        g = torch.tensor([0.1, -9.8, 0.3], device="cuda", requires_grad=True)
        xo, vo = autograd.MPMTimestep.apply(xs, vs, m, g, res, 1e-3)
        grads = torch.autograd.grad([xo, vo], [xs, vs, m], [t(pad(vals[:, 4:7], 3)), t(pad(vals[:, 7:10], 3))])
        outs.append([a.detach()[:n_near].cpu().numpy() for a in (xo, vo, *grads)])
    for a, b in zip(*outs):
        assert np.isfinite(b).all()
        assert np.abs(a - b).max() <= 8e-6 * np.abs(b).max() + 1e-9


@pytest.mark.parametrize("calls", [[1] * 11, [2] * 11, [5, 5, 3] + [5] * 8 + [3] * 7 + [5, 7] * 9, [64] * 7,
                                   ([4] * 6 + [3] * 6) * 3 + [4] * 25,
                                   [131, 146, 17, 140, 130, 17, 135, 40, 17, 133]])
@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("outer", [False, True])
def test_steps_before_and_after_their_graphs_are_made(gpu, calls, sparse, outer):
    """Call lengths repeated until a step's, a call's and the 16-step graph are
    made and used, also inside the caller's own capture (outer: every third
    call is captured and its graph launched): against launches without graphs.
    Free particles and the bounds of
    test_steps_launched_one_by_one_and_in_graphs_agree."""
    import torch

    rng = np.random.default_rng(12)
    N, n = 700, (32, 31, 30)
    dx = 1.0 / 16
    scene = gpu.Scene(n, dx, 2e-4, (0.0, 0.0, 0.0), (0.0, 0.0, 0.0), 0, 0, 0)
    st = _scene_state(rng, N, n, dx, margin=8.0)
    mats = [gpu.createElasticMaterial(1000.0, 0.0, 0.3)]
    outs = []
    for graph in (1, 0):
        sim = gpu.Simulator([scene], [N], mats, sparse_tiles=2048 if sparse else None)
        sim.set_tuning(use_graph=graph)
        sim.upload(st["x"], st["v"], st["C"], st["F"], st["m"], st["V0"])
        graphs, s = [], torch.cuda.Stream()
        for i, k in enumerate(calls):
            if outer and graph and i % 3 == 2:
                torch.cuda.synchronize()
                graphs.append(torch.cuda.CUDAGraph())
                with torch.cuda.graph(graphs[-1], stream=s):
                    sim.step(k, stream=torch.cuda.current_stream())
                graphs[-1].replay()
                torch.cuda.synchronize()
            else:
                sim.step(k)
        assert sim.status() == 0
        outs.append(sim.download())
    ulps = sum(calls) * 2.0 ** -23
    assert np.abs(outs[0]["x"] - outs[1]["x"]).max() <= 1.4 * ulps + 1e-6
    assert np.abs(outs[0]["v"] - outs[1]["v"]).max() <= (4 * ulps + 1e-6) * np.abs(outs[1]["v"]).max()


@pytest.mark.parametrize("N", [1, 31, 33, 257, 1000])
def test_downloads_of_every_subset(gpu, N):
    """Each choice of x, v, C and F comes back bit for bit, and the words around
    the arrays stay: x and v alone are stored from their planes, records with C
    or F through shared memory."""
    import itertools

    import torch
    rng = np.random.default_rng(N)
    dx = 1.0 / 32
    st = _scene_state(rng, N, (20, 24, 28), dx)
    sim = gpu.Simulator([gpu.Scene((20, 24, 28), dx, 1e-4)], [N], [gpu.createElasticMaterial(1000.0, 1e4, 0.3)])
    sim.upload(st["x"], st["v"], st["C"], st["F"], st["m"], st["V0"])
    widths = {"x": 3, "v": 3, "C": 9, "F": 9}
    for r in range(1, 5):
        for names in itertools.combinations(widths, r):
            bufs = {k: torch.full((N * widths[k] + 3,), 7.0, device="cuda") for k in names}
            sim.download({k: b[1:1 + N * widths[k]] for k, b in bufs.items()})
            torch.cuda.synchronize()
            for k, b in bufs.items():
                assert b[0] == 7.0 and torch.all(b[-2:] == 7.0)
                assert np.array_equal(b[1:1 + N * widths[k]].cpu().numpy().reshape(N, -1), st[k].reshape(N, -1)), (names, k)
