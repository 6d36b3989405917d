"""The hash grid's dense and hashed queries, and the contact coupling's cell
walk, over the forms they accept: neighbour lists are whole numbers and must be
equal; the coupling's pair count must equal a brute-force count in the
reference's float operations, and its forces are sums of at most a few hundred
pair forces taken in another order (1e-5 of the largest, as the coupling's
other tests)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,src,clustered", [((16, 16, 16), 1, False), ((13, 9, 21), 1, False), ((13, 9, 21), 2, True),
                                               ((7, 30, 5), 0, False), ((3, 2, 1), 3, False), ((61, 2, 2), 1, False),
                                               ((700, 1, 2), 1, False), ((24, 24, 24), 5, True)])
def test_dense_queries_equal_hashed_queries(gpu, res, src, clustered):
    rng = np.random.default_rng(sum(res) + src)
    cell = 0.125
    ext = np.array(res) * cell
    n = 4 * int(np.prod(res)) + 17
    pts = rng.uniform(-0.3, ext + 0.3, (n, 3))
    if clustered:
        pts[: n // 2] = ext * 0.4 + rng.normal(0, cell, (n // 2, 3))
    pts = pts.astype(np.float32)
    g = gpu.SpatialHashGrid(cell, (0.0, 0.0, 0.0), tuple(float(e) for e in ext), max_particles=n)
    assert g.resolution == tuple(res)
    g.buildHashTable(pts)
    radius = (src - 0.5) * cell if src else 0.0
    off, idx = g.neighbors(pts, radius)  # as many queries as particles: dense where buckets allow it
    assert off[0] == 0 and np.all(np.diff(off) >= 0) and off[-1] == len(idx)
    small = max(1, int(np.prod(res)) // 5)  # fewer than a query per 4 cells: hashed
    for k in range(0, n, max(small, n // 7)):
        o, i = g.neighbors(pts[k:k + small], radius)
        assert np.array_equal(o, off[k:k + small + 1] - off[k])
        assert np.array_equal(i, idx[off[k]:off[min(k + small, n)]])


def test_dense_queries_into_a_small_device_buffer_write_nothing(gpu):
    import torch
    from physgrad_b200 import _capi as C
    rng = np.random.default_rng(3)
    pts = torch.tensor(rng.random((3000, 3)).astype(np.float32), device="cuda")
    g = gpu.SpatialHashGrid(0.1, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), max_particles=3000)
    L, st, tot = gpu.lib(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.c_int64()
    C.check(L.pgmpm_hashgrid_build(g._h, pts.data_ptr(), 3000, C.PTR_DEVICE, st))
    off = torch.zeros(3001, dtype=torch.int64, device="cuda")
    out = torch.full((500000,), -7, dtype=torch.int32, device="cuda")
    for cap in (0, 10, None):
        C.check(L.pgmpm_hashgrid_neighbors(g._h, pts.data_ptr(), 3000, 0.1, off.data_ptr(), out.data_ptr(),
                                           tot.value if cap is None else cap, ctypes.byref(tot), C.PTR_DEVICE, st))
        assert tot.value == int(off[-1]) and 3000 < tot.value < 500000
        assert torch.all(out[tot.value if cap is None else 0:] == -7)
    g.n = 3000
    o, i = g.neighbors(pts.cpu().numpy(), 0.1)
    assert np.array_equal(off.cpu().numpy(), o) and np.array_equal(out[: tot.value].cpu().numpy().view(np.uint32), i)


@pytest.mark.parametrize("nodes,radius,N,Q", [(9, 0.2, 1, 1), (12, 0.3, 300, 50), (33, 0.04, 4000, 700),
                                              (33, 0.4, 900, 90), (65, 0.021, 20000, 3000)])
def test_contact_pairs_equal_brute_force(gpu, nodes, radius, N, Q):
    rng = np.random.default_rng(nodes + N)
    dx = 1.0 / (nodes - 1)
    x = rng.uniform(0.02, 0.98, (N, 3)).astype(np.float32)
    v = rng.normal(0, 0.3, (N, 3)).astype(np.float32)
    V0 = np.full(N, (dx / 2) ** 3, np.float32)
    sim = gpu.Simulator([gpu.Scene((nodes,) * 3, dx, 1e-4)], [N], [gpu.createElasticMaterial(1000.0, 1e4, 0.3)])
    sim.upload(x, v, None, None, (1000 * V0).astype(np.float32), V0)
    sx = rng.uniform(-0.05, 1.05, (Q, 3)).astype(np.float32)  # some outside the domain
    sx[0] = x[0]  # zero distance
    sv = rng.normal(0, 0.3, (Q, 3)).astype(np.float32)
    f, mf, pairs, energy = sim.sph_coupling(sx, sv, radius=radius)
    r32 = np.float32(radius)
    want_f, want_m, count, want_e = np.zeros((Q, 3)), np.zeros((N, 3)), 0, 0.0
    for q in range(Q):
        e = x - sx[q]
        d = np.sqrt((e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1]) + e[:, 2] * e[:, 2])
        near = np.flatnonzero(d < r32)
        count += len(near)
        pen = np.float64(r32) - d[near]
        want_e += 0.5e5 * (pen ** 2).sum()
        near = near[d[near] >= np.float32(1e-6)]
        e64 = x[near].astype(np.float64) - sx[q]
        dist = np.sqrt((e64 ** 2).sum(1))
        nrm, pen, dv = e64 / dist[:, None], np.float64(r32) - dist, v[near].astype(np.float64) - sv[q]
        vn = (dv * nrm).sum(1)
        t = dv - nrm * vn[:, None]
        ts = np.sqrt((t ** 2).sum(1))
        fr = np.where(ts[:, None] > 1e-6, t / np.maximum(ts, 1e-30)[:, None] * (-0.3 * 1e5 * pen)[:, None], 0.0)
        force = nrm * (1e5 * pen + 1e3 * vn)[:, None] + fr
        want_f[q] -= force.sum(0)
        np.add.at(want_m, near, force)
    assert pairs == count
    assert abs(energy - want_e) <= 1e-5 * want_e + 1e-12
    assert np.abs(f - want_f).max() <= 1e-5 * np.abs(want_f).max() + 1e-6
    assert np.abs(mf - want_m).max() <= 1e-5 * np.abs(want_m).max() + 1e-6


def test_more_cells_than_32_bits_are_refused(gpu):
    """2^22 cells an axis: their number is a multiple of 2^64, which the check
    of the whole product took for none."""
    with pytest.raises(gpu.PGMPMError, match="more than"):
        gpu.SpatialHashGrid(2.0 ** -22, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), max_particles=100)
    one = np.ones(1, np.float32)
    sim = gpu.Simulator([gpu.Scene((65,) * 3, 1.0 / 64, 1e-4)], [1], [gpu.createElasticMaterial(1000.0, 1e4, 0.3)])
    sim.upload(np.full((1, 3), 0.5, np.float32), None, None, None, one, one)
    with pytest.raises(gpu.PGMPMError, match="more than"):
        sim.sph_coupling(np.full((1, 3), 0.5, np.float32), np.zeros((1, 3), np.float32), radius=2.0 ** -22)


@pytest.mark.parametrize("res", [(16, 16, 1), (32, 32, 2), (64, 8, 8), (20, 20, 20)])
@pytest.mark.parametrize("device", [False, True])
def test_grid_order_index_longer_than_the_sort_buffers(gpu, res, device):
    """Buckets that several cells share are repeated in the grid-order index;
    with more than two entries a particle (or all particles in such a bucket)
    the first query set finds the buffers too short and takes the hashed route,
    the next ones a longer index, also after other builds.  Lists against small
    query sets, which are hashed."""
    import torch
    from physgrad_b200 import _capi as C
    rng = np.random.default_rng(sum(res))
    cell = 0.125
    ext = np.array(res) * cell
    n = max(6 * int(np.prod(res)) + 5, 20011)  # 2^19 cells to look up: not hashed for want of work
    clouds = [rng.uniform(0, ext, (n, 3)), rng.uniform(0, ext, (n, 3))]
    clouds[1][:] = clouds[1][0]  # one cell
    clouds[1][: n // 3] = rng.uniform(0, ext, (n // 3, 3))
    L, st, tot = gpu.lib(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.c_int64()
    g = gpu.SpatialHashGrid(cell, (0.0, 0.0, 0.0), tuple(float(e) for e in ext), max_particles=n)
    for build in (0, 1, 0):
        pts = clouds[build].astype(np.float32)
        # (the crowded cell's lists are long: fewer queries ask for it)
        qs = np.concatenate([pts[: n // 3], rng.uniform(0, ext, (n - n // 3, 3)).astype(np.float32)])
        g.buildHashTable(pts)
        want = [g.neighbors(qs[k:k + 20], 0.1) for k in range(0, n, n // 9)]
        for _ in range(3):
            if device:
                q = torch.tensor(qs, device="cuda")
                off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
                for cap in (0, None):  # the length, then the lists
                    idx = torch.full((tot.value if cap is None else 1,), -7, dtype=torch.int32, device="cuda")
                    C.check(L.pgmpm_hashgrid_neighbors(g._h, q.data_ptr(), n, 0.1, off.data_ptr(), idx.data_ptr(),
                                                       idx.numel() if cap is None else 0, ctypes.byref(tot),
                                                       C.PTR_DEVICE, st))
                off, idx = off.cpu().numpy(), idx.cpu().numpy().view(np.uint32)
            else:
                off, idx = g.neighbors(qs, 0.1)
            assert off[-1] == len(idx)
            for (o, i), k in zip(want, range(0, n, n // 9)):
                assert np.array_equal(o, off[k:k + len(o)] - off[k])
                assert np.array_equal(i, idx[off[k]:off[k] + len(i)])


@pytest.mark.parametrize("res,src,clustered", [((16, 16, 16), 1, False), ((13, 9, 21), 1, True), ((13, 9, 21), 2, True),
                                               ((7, 30, 5), 0, False), ((3, 2, 1), 3, False), ((1, 1, 1), 1, False),
                                               ((61, 2, 2), 1, False), ((700, 1, 2), 1, False), ((9, 9, 9), 5, False)])
@pytest.mark.parametrize("more_queries_than_particles", [False, True])
def test_many_queries_on_small_grids_equal_hashed_queries(gpu, res, src, clustered, more_queries_than_particles):
    """Enough queries for the grid-order tables on grids of few cells and odd
    shapes, inside the grid and outside, in the sort's buffers and in their
    own: offsets and lists against small query sets, which are hashed."""
    rng = np.random.default_rng(sum(res) + 7 * src)
    cell = 0.125
    ext = np.array(res) * cell
    nq = -(-(1 << 19) // (2 * src + 1) ** 3) + 3
    n = min(nq, 2 * int(np.prod(res)) + 9)
    cap = n if more_queries_than_particles else nq
    pts = rng.uniform(-0.3, ext + 0.3, (n, 3))
    if clustered:
        pts[: n // 2] = ext * 0.4 + rng.normal(0, cell, (n // 2, 3))
    qs = rng.uniform(-0.3, ext + 0.3, (nq, 3)).astype(np.float32)
    g = gpu.SpatialHashGrid(cell, (0.0, 0.0, 0.0), tuple(float(e) for e in ext), max_particles=cap)
    assert g.resolution == tuple(res)
    g.buildHashTable(pts.astype(np.float32))
    radius = (src - 0.5) * cell if src else 0.0
    off, idx = g.neighbors(qs, radius)
    assert off[0] == 0 and np.all(np.diff(off) >= 0) and off[-1] == len(idx)
    part = min(nq // 8, 300)
    for k in (0, nq // 3, nq - part):
        o, i = g.neighbors(qs[k:k + part], radius)
        assert np.array_equal(o, off[k:k + part + 1] - off[k])
        assert np.array_equal(i, idx[off[k]:off[k + part]])


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 4097, (1 << 18) - 1, 1 << 18, (1 << 18) + 1, (1 << 18) + 4097])
def test_counts_scanned_at_the_edges_of_blocks_and_rows(gpu, n):
    """The exclusive scan takes one or four rows a warp by the number of counts:
    offsets of n queries and the starts of n cells against numpy's sums."""
    rng = np.random.default_rng(n)
    pts = rng.uniform(0, 1, (500, 3))
    pts[:, 0] *= n  # n cells in a row
    g = gpu.SpatialHashGrid(1.0, (0.0, 0.0, 0.0), (float(n), 1.0, 1.0), max_particles=700)
    assert g.total_cells == n
    g.buildHashTable(pts.astype(np.float32))
    counts, starts = g.getCellParticleCounts().astype(np.int64), g.getCellStartIndices()
    assert counts.sum() == 500 and np.array_equal(starts, np.concatenate([[0], np.cumsum(counts)[:-1]]))
    qs = rng.uniform(0, 1, (n, 3)) * [n, 1, 1]
    off, idx = g.neighbors(qs.astype(np.float32), 0.0)
    assert off[0] == 0 and off[-1] == len(idx) and np.all(np.diff(off) >= 0)
    for k in np.unique(np.concatenate([[0, n - 1], rng.integers(0, n, 40)])):
        o, i = g.neighbors(qs[k:k + 1].astype(np.float32), 0.0)
        assert o[1] == off[k + 1] - off[k] and np.array_equal(i, idx[off[k]:off[k + 1]])
