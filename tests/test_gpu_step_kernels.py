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
