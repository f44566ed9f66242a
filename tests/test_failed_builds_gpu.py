"""Builds that fail, and what a caller may do after them.  Every allocation that
is refused here is larger than the device, so the device keeps its memory."""
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


def test_a_call_of_no_steps_after_a_failed_one(gpu_pkg):
    """66,000 particles crowd into reach of each other: their rows fit, the
    pair list (past 2^31) does not, and the step is refused between the two.  A
    call of no steps then sums W over the rows."""
    N, H = 66000, 0.01
    rng = np.random.default_rng(8)
    x = 0.05 + 0.9 * rng.random((2, N))
    c = gpu_pkg.GPUCellList(tuple(x), (H, H), H, MIN=(0.0, 0.0), MAX=(1.0, 1.0))
    h = H / 2
    prob = gpu_pkg.SPHProblem(c, h / 1.5, h, H, gpu_pkg.WendlandC2(dim=2), np.full(N, 1000.0), np.full(N, 2, np.int32),
                              1000.0, 1.0, 1e-6, 0.01, 40.0, 7, 0.1, 0.2)
    prob.set_lanes(4)
    y = 0.5005 + 0.2 * H * rng.random((2, N))  # one cell
    for d in range(2):
        c.points[d].copy_(torch.from_numpy(y[d]))
    with pytest.raises(gpu_pkg.GcsphError) as e:
        prob.stepsolve(1)
    assert e.value.code == gpu_pkg._lib.GCSPH_ECAPACITY
    assert prob.stepsolve(0)[0] == 0
    got = prob.field("sumW").cpu().numpy()
    for i in (0, 1234, N - 1):
        u = np.delete(np.hypot(y[0] - y[0, i], y[1] - y[1, i]), i) / H
        want = (7.0 / np.pi / H**2) * ((1.0 + 4.0 * u) * (1.0 - u) ** 4).sum()
        # a sum of N positive terms: N roundings of it at the very most
        assert abs(got[i] - want) <= N * 2.0**-52 * want
