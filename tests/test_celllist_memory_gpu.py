"""What the cell list's search keeps between update! and its emit, in bytes:
no more than four a pair (the neighbours of all points in one array) and a row
of 256 a point, whatever the points' distribution over the cells."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _used():
    """Device memory in use outside torch's own pool."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    return total - free - torch.cuda.memory_reserved()


SLACK = 16 << 20  # the allocator's granularity


def test_points_that_crowd(gpu_pkg):
    """20,000 points of one cell come into reach of each other: 10,000 pairs a
    point in the mean, twice that at the most."""
    N, dist = 20000, 1e-3
    x = 0.01 + 0.9 * np.random.default_rng(4).random((2, N))
    c = gpu_pkg.GPUCellList(tuple(x), (1.0, 1.0), dist, MIN=(0.0, 0.0), MAX=(1.0, 1.0), mpairs=100_000)
    before = _used()
    for p in c.points:
        p.mul_(1e-4)
    c.update()
    assert c.pairsn == N * (N - 1) // 2
    assert _used() - before <= 4 * (c.pairsn + 256 * N) + SLACK


def test_cells_wider_than_the_reach(gpu_pkg):
    """Thousands of candidates a point of which hardly any is a pair."""
    N, dist = 300000, 1e-3
    x = np.random.default_rng(6).random((2, N))
    before = _used()
    c = gpu_pkg.GPUCellList(tuple(x), (0.1, 0.1), dist, MIN=(0.0, 0.0), MAX=(1.0, 1.0), mpairs=400_000)
    assert 0 < c.pairsn < N
    # next to the positions and indices that any list of N points holds
    assert _used() - before <= 4 * (c.pairsn + 256 * N) + SLACK


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("N", [6000, 60000])
def test_a_uniform_set_is_searched_once(gpu_pkg, D, N):
    """The first search's guess of what a point keeps holds: the construction
    launches what an update! does, and no second search (20 pairs a point)."""
    x = np.random.default_rng(N + D).random((D, N))
    ball = np.pi if D == 2 else 4.0 * np.pi / 3.0
    dist = (40.0 / (N * ball)) ** (1.0 / D)
    n0 = gpu_pkg.launch_count()
    c = gpu_pkg.GPUCellList(tuple(x), (dist,) * D, dist, MIN=(0.0,) * D, MAX=(1.0,) * D, mpairs=22 * N)
    n1 = gpu_pkg.launch_count()
    c.update()
    assert n1 - n0 == gpu_pkg.launch_count() - n1
