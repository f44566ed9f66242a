"""Builds that fail for want of memory, and what a caller may do after them:
every request here is larger than the device, so it is refused at once and the
device keeps its memory."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _spread(pkg):
    """420,000 points of one cell, few of them in reach of each other; closer()
    brings all of them within it, and what a search would keep of them then
    (353 GB and more) is refused."""
    N, dist = 420000, 1e-3
    x = 0.01 + 0.9 * np.random.default_rng(4).random((2, N))
    c = pkg.GPUCellList(tuple(x), (1.0, 1.0), dist, MIN=(0.0, 0.0), MAX=(1.0, 1.0), mpairs=1_000_000)
    home = [p.clone() for p in c.points]

    def closer():
        for p in c.points:
            p.mul_(1e-4)

    def back():
        for p, q in zip(c.points, home):
            p.copy_(q)
    return c, closer, back


def test_a_refused_allocation_is_reported_once(gpu_pkg):
    """update! reports it; the calls after it, torch's and the library's, run."""
    c, closer, back = _spread(gpu_pkg)
    before = c.neighborlistview().clone()
    closer()
    with pytest.raises(gpu_pkg.GcsphError) as e:
        c.update()
    assert e.value.code == gpu_pkg._lib.GCSPH_ENOMEM
    back()
    d, _, _ = _spread(gpu_pkg)
    assert torch.equal(d.neighborlistview(), before)


def test_a_failed_partialupdate_leaves_no_list(gpu_pkg):
    """The list from before is overwritten by then: none is handed out, and
    the next update! makes one again."""
    c, closer, back = _spread(gpu_pkg)
    before = c.neighborlistview().clone()
    closer()
    with pytest.raises(gpu_pkg.GcsphError) as e:
        c.partialupdate()
    assert e.value.code == gpu_pkg._lib.GCSPH_ENOMEM
    L, n = gpu_pkg.load_library(), C.c_int64(-1)
    # (asks for the count alone: nothing is launched)
    assert L.gcl_emit_pairs(c._h, None, 0, 0, C.byref(n)) == gpu_pkg._lib.GCSPH_ESTATE
    back()
    c.update()
    assert torch.equal(c.neighborlistview(), before)
