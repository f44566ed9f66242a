"""Captured steps hold the addresses of the cell list's buffers: a graph from
before one of them moved is not replayed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _last_call_captures(pkg, scale):
    """Graphs that the last of these calls captures: a step (captured and
    replayed), three steps with the points closer by `scale`, and the first
    kind again with the points back."""
    dx = 0.01
    g = np.arange(60) * dx + 0.2
    x = np.stack([a.ravel() for a in np.meshgrid(g, g, indexing="ij")])
    x = x + np.random.default_rng(3).uniform(-0.1, 0.1, x.shape) * dx
    N, H = x.shape[1], 3.38 * dx
    c = pkg.GPUCellList(tuple(x), (H, H), H, MIN=(0.0, 0.0), MAX=(1.0, 1.0))
    prob = pkg.SPHProblem(c, dx, H / 2, H, pkg.WendlandC2(dim=2), np.full(N, 1000.0), np.full(N, 2, np.int32),
                          1000.0, 0.1, 1e-7, 0.01, 40.0, 7, 0.1, 0.2)
    prob.set_lanes(4)
    c.update()
    n0 = c.pairsn
    for _ in range(2):
        prob.stepsolve(1)
    assert prob.graph_stats() == (1, 1)
    where = [p.clone() for p in c.points]
    for p in c.points:
        p.mul_(scale)
    c.update()
    assert c.pairsn < 1.25 * n0  # the neighbour rows' buffer stays
    dense = 2 * c.pairsn / N
    prob.stepsolve(3)
    for p, q in zip(c.points, where):
        p.copy_(q)
    c.update()
    before = prob.graph_stats()[0]
    prob.stepsolve(1)
    return prob.graph_stats()[0] - before, 2 * n0 / N, dense


def test_staged_rows_that_outgrow_their_buffer(gpu_pkg):
    """Rows are staged 64 entries wide up to 37.3 neighbours a point and 128 from
    there on; the buffer moves when they widen."""
    captured, _, _ = _last_call_captures(gpu_pkg, 1.0)
    assert captured == 0
    captured, sparse, dense = _last_call_captures(gpu_pkg, 0.93)
    assert sparse < 37.3 < dense
    assert captured == 1
