"""Calls that fail among a step's launches, and what the next call finds.

The failures are made on the host: a preloaded stand-in for the launch entry
of the CUDA runtime returns an error for the k-th launch without launching
(child processes), or an error is left pending in the thread.  Two runs of
one state differ by FP32 summation order: x <= 1e-6 absolute, v <= 1e-4 of
the largest, F <= 1e-5, as in test_gpu_step_kernels.py.
"""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static int launch_left = 0, build_left = 0;
void fail_launch(int k) { launch_left = k; }   /* the k-th launch from now fails; 0: none */
void fail_builds(int k) { build_left = k; }    /* the next k graph instantiations fail */
static void* real(const char* name) {
    return dlsym(dlopen("libcudart.so.12", RTLD_NOLOAD | RTLD_LAZY), name);
}
int cudaLaunchKernelExC(const void* cfg, const void* f, void** args) {
    static int (*next)(const void*, const void*, void**) = NULL;
    if (!next) next = (int (*)(const void*, const void*, void**))real("cudaLaunchKernelExC");
    if (launch_left > 0 && --launch_left == 0) return 701; /* cudaErrorLaunchOutOfResources */
    return next(cfg, f, args);
}
static int alloc_left = 0;
void fail_allocs(int k) { alloc_left = k; }      /* the next k allocations fail */
static size_t no_alloc = 0;
void fail_alloc(size_t bytes) { no_alloc = bytes; }  /* allocations of this size fail; 0: none */
int cudaMalloc(void** p, size_t bytes) {
    static int (*next)(void**, size_t) = NULL;
    if (!next) next = (int (*)(void**, size_t))real("cudaMalloc");
    if (alloc_left > 0) {
        --alloc_left;
        return 2; /* cudaErrorMemoryAllocation */
    }
    return no_alloc && bytes == no_alloc ? 2 : next(p, bytes);
}
int cudaGraphInstantiate(void** exec, void* graph, unsigned long long flags) {
    static int (*next)(void**, void*, unsigned long long) = NULL;
    if (!next) next = (int (*)(void**, void*, unsigned long long))real("cudaGraphInstantiate");
    if (build_left > 0) {
        --build_left;
        return 2; /* cudaErrorMemoryAllocation */
    }
    return next(exec, graph, flags);
}
"""

COMMON = r"""
import ctypes, sys
import numpy as np
import physgrad_b200 as pg
from physgrad_b200 import _capi as C, workloads as W
shim = ctypes.CDLL(None)

def close(a, b):
    assert np.abs(a["x"] - b["x"]).max() <= 1e-6
    assert np.abs(a["v"] - b["v"]).max() <= 1e-4 * np.abs(b["v"]).max() + 1e-7
    assert np.abs(a["F"] - b["F"]).max() <= 1e-5

def raises(fn):
    try:
        fn()
    except Exception as e:
        return True
    return False

scenes, counts, mats, st, _ = W.elastic_cube(n_particles=3000, n=24, v_sigma=0.5, seed=5)
N = counts[0]
def solver():
    return pg.Simulator(scenes, counts, mats, sparse_tiles=512 if SPARSE else None)
def upload(s):
    s.upload(st["x"], st["v"], None, None, st["m"], st["V0"])
fresh = solver()
upload(fresh)
fresh.step(5)
want = fresh.download()
"""

STEPS = COMMON + r"""
sim = solver()
sim.set_tuning(use_graph=0)
failed = 0
for k in range(1, 17):  # 6 + 5 + 5 launches
    upload(sim)
    shim.fail_launch(k)
    failed += raises(lambda: sim.step(3))
    shim.fail_launch(0)
    before = sim.get_array(C.ARRAY_KEYS)
    sim.step(1)
    order = sim.get_array(C.ARRAY_SORTED_ORDER)
    assert np.array_equal(np.sort(order), np.arange(N)), k
    assert np.array_equal(before[order], np.sort(before)), k
    upload(sim)
    sim.step(5)
    assert sim.status() == 0
    close(sim.download(), want)
assert failed == 16, failed
print("CHILD OK")
"""

PIC = r"""
import ctypes
import numpy as np, torch
from physgrad_b200.autograd import MPMTimestep
shim = ctypes.CDLL(None)
rng = np.random.default_rng(3)
N, res = 3000, 32
t = lambda a: torch.tensor(a.astype(np.float32), device="cuda")
x, v, m, g = t(rng.uniform(0.2, 0.8, (N, 3))), t(rng.normal(0, 1, (N, 3))), t(rng.uniform(0.5, 1.5, N)), t(np.array([0, -9.8, 1]))
gx, gv = t(rng.normal(0, 1, (N, 3))), t(rng.normal(0, 1, (N, 3)))
for a in (x, v, m, g):
    a.requires_grad_(True)
def step(fwd=0, bwd=0):
    torch.cuda.synchronize()
    shim.fail_launch(fwd)
    xo, vo = MPMTimestep.apply(x, v, m, g, res, 1e-3)
    shim.fail_launch(bwd)
    gr = torch.autograd.grad([xo, vo], [x, v, m, g], [gx, gv])
    shim.fail_launch(0)
    return [a.detach().cpu().numpy() for a in (xo, vo, *gr)]
want = step()
failed = 0
for k in range(1, 7):  # 6 launches each way
    for way in ({"fwd": k}, {"bwd": k}):
        try:
            step(**way)
        except Exception:
            failed += 1
        shim.fail_launch(0)
        for a, b in zip(step(), want):
            assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max(), (k, way)
assert failed == 12, failed
print("CHILD OK")
"""


BUILDS = COMMON + r"""
direct = solver()
direct.set_tuning(use_graph=0)
sim = solver()
shim.fail_builds(1000)
for calls in ([5] * 7, [1] * 10, [140] * 6):
    for s in (sim, direct):
        upload(s)
        for k in calls:
            s.step(k)
    assert sim.status() == direct.status() == 0
    assert pg.lib().pgmpm_last_error() == b""
    if calls[0] < 100:  # (longer runs drift apart by rounding)
        close(sim.download(), direct.download())
shim.fail_builds(0)
sim.set_tuning(use_graph=1)
upload(sim)
for _ in range(7):
    sim.step(5)
upload(sim)
sim.step(5)
close(sim.download(), want)
print("CHILD OK")
"""

BACKWARD = COMMON + r"""
shim.fail_alloc.argtypes = [ctypes.c_size_t]
rng = np.random.default_rng(9)
go = {k: rng.normal(0, 1, (N, d)).astype(np.float32) for k, d in (("x", 3), ("v", 3), ("C", 9), ("F", 9))}
def grads(s, no_alloc=0):
    upload(s)
    s.forward_checkpointed(9, 4)
    shim.fail_alloc(no_alloc)
    g = s.backward(go)
    shim.fail_alloc(0)
    return g
want = grads(solver())
sim = solver()
for size in (64 * N, 0):  # without memory for the scatter's payload, then with it
    for _ in range(2):
        got = grads(sim, size)
        for k in want:
            a, b = np.asarray(got[k]), np.asarray(want[k])
            assert np.abs(a - b).max() <= 1e-4 * np.abs(b).max(), k
    assert sim.status() == 0
print("CHILD OK")
"""

HASH = COMMON + r"""
rng = np.random.default_rng(4)
pts = rng.uniform(0, 1, (20011, 3)).astype(np.float32)
grid = lambda: pg.SpatialHashGrid(0.07, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), max_particles=len(pts))
a = grid()
shim.fail_allocs(1)
b = grid()  # without the tables of the dense queries
shim.fail_allocs(2)
assert raises(grid)
shim.fail_allocs(0)
a.buildHashTable(pts)
b.buildHashTable(pts)
for _ in range(2):
    (oa, ia), (ob, ib) = a.neighbors(pts, 0.07), b.neighbors(pts, 0.07)
    assert np.array_equal(oa, ob) and np.array_equal(ia, ib)
# a bucket of its own for nearly all particles: more entries than the sort's
# buffers hold, and no memory for a longer index
c = grid()
pts[: len(pts) - 100] = pts[0]
c.buildHashTable(pts)
b.buildHashTable(pts)
qs = rng.uniform(0, 1, (20011, 3)).astype(np.float32)
want = b.neighbors(qs, 0.07)
for k in (0, 1, 0):
    shim.fail_allocs(k)
    L, tot = pg.lib(), ctypes.c_int64()
    got = c.neighbors(qs, 0.07) if not k else None
    if k:  # into arrays that are there (host staging is)
        off, idx = np.zeros(len(qs) + 1, np.int64), np.zeros(len(want[1]), np.uint32)
        assert L.pgmpm_hashgrid_neighbors(c._h, qs.ctypes.data, len(qs), 0.07, off.ctypes.data, idx.ctypes.data, len(idx),
                                          ctypes.byref(tot), C.PTR_HOST, None) == 0
        got = off, idx
    shim.fail_allocs(0)
    assert np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1])
print("CHILD OK")
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("shim")
    (d / "shim.c").write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(d / "shim.so"), str(d / "shim.c"), "-ldl"], check=True)
    return str(d / "shim.so")


def _child(shim, code):
    env = dict(os.environ, LD_PRELOAD=shim, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "CHILD OK" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]


@pytest.mark.parametrize("sparse", [False, True])
def test_steps_after_a_call_that_failed_between_launches(gpu, shim, sparse):
    """A three-step call whose k-th launch fails, for every k: the next step
    sorts each particle once (a step's G2P counts the next step's keys, which a
    failed call leaves counted), and after an upload five steps are those of a
    fresh solver."""
    _child(shim, f"SPARSE = {sparse}\n" + STEPS)


def test_pic_steps_after_a_call_that_failed_between_launches(gpu, shim):
    """The same for each launch of the PIC step's forward and backward."""
    _child(shim, PIC)


def test_steps_whose_graphs_cannot_be_made(gpu, shim):
    """Every graph instantiation fails for want of memory: the steps run
    kernel by kernel, no call fails, and graphs are made again afterwards."""
    _child(shim, "SPARSE = False\n" + BUILDS)


def test_backward_without_memory_for_the_scatter_payload(gpu, shim):
    """The reverse pass needs 64 bytes per particle more for the scatter's
    payload only where they are to be had: gradients with and without it agree
    (sums of FP32 terms in another order, the bound of the other reverse
    scatters' comparison on a whole rollout)."""
    _child(shim, "SPARSE = False\n" + BACKWARD)


def test_hash_grid_without_memory_for_the_dense_queries(gpu, shim):
    """A grid whose tables cannot be had answers by the hashed queries, as one
    whose index in grid order cannot grow; without memory for the rest its
    creation fails.  Lists are whole numbers and equal."""
    _child(shim, "SPARSE = False\n" + HASH)


def test_steps_with_an_error_pending_in_the_thread(gpu):
    """An error that an earlier CUDA call of the thread left pending is not
    taken for a step's own, and a create that runs out of memory leaves none."""
    from physgrad_b200 import PGMPMError
    from physgrad_b200 import workloads as W

    rt = ctypes.CDLL("libcudart.so.12")
    scenes, counts, mats, st, _ = W.elastic_cube(n_particles=3000, n=24, v_sigma=0.5, seed=5)
    outs = []
    for pending in (False, True):
        sim = gpu.Simulator(scenes, counts, mats)
        sim.upload(st["x"], st["v"], None, None, st["m"], st["V0"])
        if pending:
            with pytest.raises(PGMPMError):  # 206 GB of state planes
                gpu.Simulator(scenes, [2 ** 31 - 16], mats)
            assert rt.cudaPeekAtLastError() == 0
            assert rt.cudaSetDevice(4096) != 0 and rt.cudaPeekAtLastError() != 0
        sim.step(5)
        rt.cudaGetLastError()
        assert sim.status() == 0
        outs.append(sim.download())
    assert np.abs(outs[0]["x"] - outs[1]["x"]).max() <= 1e-6
    assert np.abs(outs[0]["v"] - outs[1]["v"]).max() <= 1e-4 * np.abs(outs[0]["v"]).max()
