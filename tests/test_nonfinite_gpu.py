"""Infinities and NaN in a state: split rows (a group of lanes a particle) give
what serial rows give, which are the oracle's to the bit -- a diverged run is
reported by the same particles whatever form its size picks."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "v", "x", "P", "a", "drhodt", "rhoh", "vh", "xh", "cdx", "sumW", "sumgW", "buf2")


def _case(pkg, D, big=False, skin=1.0):
    """A tank off the lattice, walls of three kinds; `big`: more pairs than the
    pair passes have threads."""
    if D == 2:
        c = pkg.workloads.dam_break_2d(dx=0.0156 if big else 0.05, layer_ptype=(1, 1, 1))
    else:
        size = dict(fluid=(0.5, 0.6, 0.4), tank=(1.0, 0.8, 0.6)) if big else dict(fluid=(0.2, 0.3, 0.2),
                                                                                 tank=(0.4, 0.4, 0.3))
        c = pkg.workloads.dam_break_3d(dx=0.05, layer_ptype=(1, 1, 1), full_physics=False, **size)
    rng = np.random.default_rng(5)
    c.x = c.x + rng.uniform(-0.2, 0.2, c.x.shape) * c.dx
    c.rho = c.rho + rng.uniform(0.0, 2.0, c.N)
    c.dist = skin * c.H
    c.cellsize = (c.dist,) * D
    c.v = rng.uniform(-0.05, 0.05, c.x.shape)
    c.v[:, c.ptype <= 1] = 0.0
    return c


def _run(pkg, c, lanes, steps=1, **params):
    system = pkg.GPUCellList(tuple(c.x), c.cellsize, c.dist)
    prob = pkg.SPHProblem(system, c.dx, c.h, c.H, pkg.WendlandC2(dim=c.D), c.rho, c.ptype, c.rho0, c.m0, c.dt, c.alpha,
                          c.c0, c.gamma, c.delta, c.CFL, v=tuple(c.v), s=params.pop("s", 0.0))
    for k, val in params.items():
        setattr(prob, k, val)
    prob.set_lanes(lanes)
    prob.stepsolve(steps)
    out = {}
    for f in FIELDS:
        t = {"x": prob.system.points, "rho": prob.rho, "v": prob.v}.get(f)
        t = prob.field(f) if t is None else t
        out[f] = (torch.stack(t) if isinstance(t, tuple) else t).cpu().numpy()
    return out


def _same(got, want, fields=FIELDS):
    """The same particles not finite; where finite, the FP64 contract."""
    for f in fields:
        fine = np.isfinite(want[f])
        assert np.array_equal(np.isfinite(got[f]), fine), f
        if fine.any():
            assert np.abs(got[f][fine] - want[f][fine]).max() <= 1e-12 * np.abs(want[f][fine]).max(), f


def _behind_the_walls(c):
    """A wall particle with no fluid within 2 H."""
    fl = c.x[:, c.ptype > 1]
    far = [i for i in np.flatnonzero(c.ptype == 1)
           if np.sqrt(((fl - c.x[:, i:i + 1]) ** 2).sum(0)).min() > 2.0 * c.H]
    return far[len(far) // 2]


@pytest.mark.parametrize("D", [2, 3])
def test_an_infinite_density_in_cspmcorr(gpu_pkg, D):
    """It adds W m0/∞ = 0 to its neighbours' sums (a wall's, whose density the
    step itself leaves alone)."""
    c = _case(gpu_pkg, D)
    i = _behind_the_walls(c)
    c.rho[i] = np.inf
    want = _run(gpu_pkg, c, 1, cspmn=1)
    near = np.sqrt(((c.x - c.x[:, i:i + 1]) ** 2).sum(0)) < c.H
    assert near.sum() > 4 and np.isfinite(np.delete(want["rho"], i)).all()
    for lanes in (2, 4, 32):
        _same(_run(gpu_pkg, c, lanes, cspmn=1), want, ("rho", "P"))


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("val", [np.nan, np.inf])
def test_sums_over_a_diverged_particle(gpu_pkg, D, val):
    """A wall particle's velocity moves it out of the world within the step; the
    closing sums still go over the pairs that it had.  Then a call of no steps
    over the caller's points, one of them moved away by hand."""
    c = _case(gpu_pkg, D)
    i = _behind_the_walls(c)
    c.v[0, i] = val
    want = _run(gpu_pkg, c, 1)
    bad = ~np.isfinite(want["sumgW"])
    assert bad.any() and np.isfinite(want["sumW"]).all()
    c2 = _case(gpu_pkg, D)
    sums = {}
    for lanes in (1, 2, 4, 32):
        if lanes > 1:
            _same(_run(gpu_pkg, c, lanes), want, ("sumW", "sumgW"))
        system = gpu_pkg.GPUCellList(tuple(c2.x), c2.cellsize, c2.dist)
        prob = gpu_pkg.SPHProblem(system, c2.dx, c2.h, c2.H, gpu_pkg.WendlandC2(dim=D), c2.rho, c2.ptype, c2.rho0,
                                  c2.m0, c2.dt, c2.alpha, c2.c0, c2.gamma, c2.delta, c2.CFL)
        prob.set_lanes(lanes)
        system.points[1][i] = val
        prob.stepsolve(0)
        sums[lanes] = {"sumW": prob.field("sumW").cpu().numpy(),
                       "sumgW": torch.stack(prob.field("sumgW")).cpu().numpy()}
        assert not np.isfinite(sums[1]["sumgW"]).all()
        _same(sums[lanes], sums[1], ("sumW", "sumgW"))


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("field", ["rho", "v"])
@pytest.mark.parametrize("val", [np.nan, np.inf])
def test_pairs_in_the_skin(gpu_pkg, D, field, val):
    """Pairs past every term's reach add 0 at any finite state, and NaN with a
    particle that is not: the list's length picks how they are told apart."""
    c = _case(gpu_pkg, D, big=True, skin=1.2)
    fl = np.flatnonzero(c.ptype > 1)
    i = fl[len(fl) // 2]
    if field == "rho":
        c.rho[i] = val
    else:
        c.v[0, i] = val
    want = _run(gpu_pkg, c, 1, cspmn=15, nui=0.0)
    r = np.sqrt(((c.x - c.x[:, i:i + 1]) ** 2).sum(0))
    skin = (r > 1.02 * c.H) & (r < c.dist) & (c.ptype > 0)
    assert skin.sum() > 4 and not np.isfinite(want["a"][:, skin]).all(0).any()
    _same(_run(gpu_pkg, c, 4, cspmn=15, nui=0.0), want)
