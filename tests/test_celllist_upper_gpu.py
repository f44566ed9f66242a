"""The cell list's own search and its two emits, pairs and order: rows of
exactly 32 candidates and their neighbours, few and many pairs a point, a
crowded cell whose points outgrow what is kept (searched again in the emit), a
first build against later ones, moved points on stale
cells, lists cut by their capacity.  The list is exactly the oracle's pair set
ordered by (rank of the first, rank of the second), ranks by (cell, index)."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _expected(orc, x, dist, cells_of=None):
    D = x.shape[0]
    cs, off, cell = orc.grid(cells_of if cells_of is not None else x, (dist,) * D, dist)
    pcell, _ = orc.cellmap(cells_of if cells_of is not None else x, cs, off, cell)
    pairs, n = orc.neib_search(x, pcell, cell, dist)
    p = np.asarray(pairs)[:n].astype(np.int64) - 1
    pc = np.asarray(pcell).reshape(D, -1) if np.asarray(pcell).shape[0] == D else np.asarray(pcell).reshape(-1, D).T
    lin = pc[0].astype(np.int64)
    stride = 1
    for d in range(1, D):
        stride *= int(cell[d - 1])
        lin = lin + pc[d].astype(np.int64) * stride
    rank = np.empty(x.shape[1], np.int64)
    rank[np.lexsort((np.arange(x.shape[1]), lin))] = np.arange(x.shape[1])
    r = np.sort(rank[p], axis=1)
    return np.sort(p + 1, axis=1)[np.lexsort((r[:, 1], r[:, 0]))]


def _points(kind, D, N, seed):
    rng = np.random.default_rng(seed)
    x = rng.random((D, N))
    if kind == "cluster":  # a crowded cell in a sparse set
        m = N // 5
        x[:, :m] = 0.5 + 0.002 * rng.random((D, m))
    if kind == "runs":  # cells of 32 points, their neighbours of 31 and 33
        c = np.repeat(np.arange(3), [31, 32, 33])
        x = 0.05 * rng.random((D, c.size))
        x[0] += c
        x[:, 0] = 0.0
    return np.ascontiguousarray(x)


@pytest.mark.parametrize("kind,D,N,dist", [
    ("runs", 2, 0, 1.0), ("runs", 3, 0, 1.0),
    ("uniform", 2, 1, 0.1), ("uniform", 2, 257, 0.03), ("uniform", 2, 5000, 0.1), ("uniform", 2, 70001, 0.01),
    ("uniform", 3, 255, 0.3), ("uniform", 3, 9001, 0.04), ("uniform", 3, 9001, 0.2),
    ("cluster", 2, 3000, 0.02), ("cluster", 3, 3000, 0.05)])
def test_ordered_list(gpu_pkg, orc, kind, D, N, dist):
    x = _points(kind, D, N, 7 + D)
    c = gpu_pkg.GPUCellList(tuple(x), (dist,) * D, dist)
    want = _expected(orc, x, dist)
    assert np.array_equal(c.neighborlistview().cpu().numpy(), want)  # first build
    c.update()
    assert np.array_equal(c.neighborlistview().cpu().numpy(), want)
    # a list cut by its capacity, 8-byte aligned and not
    L = gpu_pkg.load_library()
    cap, n = max(1, c.pairsn // 2), C.c_int64()
    for shift in (0, 1):
        raw = torch.full((2 * cap + 3,), -7, dtype=torch.int32, device="cuda")
        L.gcl_emit_pairs(c._h, C.c_void_p(raw.data_ptr() + 4 * shift), cap, 0, C.byref(n))
        m = min(cap, c.pairsn)
        assert n.value == c.pairsn
        assert np.array_equal(raw[shift:shift + 2 * m].view(m, 2).cpu().numpy(), want[:m])
        assert int(raw[shift + 2 * m]) == -7
    # moved points on the cells as they were
    y = x + 0.3 * dist * (np.random.default_rng(5).random(x.shape) - 0.5)
    for d in range(D):
        c.points[d].copy_(torch.from_numpy(np.ascontiguousarray(y[d])))
    c.pairs = torch.zeros((4 * c.pairsn + 64, 2), dtype=torch.int32, device="cuda")
    c.partialupdate()
    assert np.array_equal(c.neighborlistview().cpu().numpy(), _expected(orc, y, dist, cells_of=x))


def test_crowding_between_updates(gpu_pkg, orc):
    """Words kept for a sparse set, then all points move into a few cells:
    the next search keeps rows, and enough of them."""
    D, N, dist = 2, 2000, 0.02
    x = _points("uniform", D, N, 3)
    c = gpu_pkg.GPUCellList(tuple(x), (dist,) * D, dist, MIN=(0, 0), MAX=(1, 1))
    c.update()
    y = np.ascontiguousarray(0.4 + 0.06 * x)
    for d in range(D):
        c.points[d].copy_(torch.from_numpy(y[d]))
    cs, off, cell = orc.grid(y, (dist,) * D, dist, (0, 0), (1, 1))
    pcell, _ = orc.cellmap(y, cs, off, cell)
    pairs, n = orc.neib_search(y, pcell, cell, dist)
    for _ in range(2):
        c.update()
        assert c.pairsn == n
        assert np.array_equal(orc.pair_set(c.neighborlistview().cpu().numpy()), orc.pair_set(pairs))
