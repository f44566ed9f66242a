"""The pair-once passes on split rows, where their pair classes and lane
counts can go wrong: walls whose pairs add nothing, walls of negative ptype
(pressure between two of them, no other term), mixed pairs within and beyond
r₀, surface tension over the whole range of its cosine, and every lane count
of the row sums.  Against the CPU oracle with the FP64 contract (1e-12
normwise, or 16x the noise of the reference's own re-ordered sums)."""
import numpy as np
import pytest

from test_sph_gpu import check, make_pair, run_both, well_conditioned_v

pytestmark = pytest.mark.gpu


def _case(pkg, D, layers):
    if D == 2:
        case = pkg.workloads.dam_break_2d(dx=0.04, fluid=(0.6, 0.8), tank=(1.2, 1.0), layer_ptype=layers)
    else:
        case = pkg.workloads.dam_break_3d(dx=0.05, fluid=(0.3, 0.4, 0.2), tank=(0.6, 0.6, 0.3), layer_ptype=layers)
    case.s = 0.05
    case.extra = dict(nu=0.2, xsph_eps=0.5, cspmn=3)
    # off the lattice, so that no separation sits at a cut
    rng = np.random.default_rng(11)
    fl = case.ptype > 1
    case.x = case.x.copy()
    case.x[:, fl] += rng.uniform(-0.05, 0.05, (D, int(fl.sum()))) * case.dx
    case.rho = case.rho + rng.uniform(0.0, 2.0, case.rho.size)
    return case


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("layers", [(1, 0, 0), (1, -1, -1), (0, -1, 1)])
@pytest.mark.parametrize("lanes", [2, 4, 32])
def test_pair_classes(gpu_pkg, orc, D, layers, lanes):
    case = _case(gpu_pkg, D, layers)
    v = well_conditioned_v(case)
    prob, ref = make_pair(gpu_pkg, orc, case, lanes, v=v)
    for _ in range(2):  # the second call replays the captured graph
        run_both(prob, ref, 4)
    check(orc, prob, ref, case, lanes, [(4, {}), (4, {})], v=v)


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("lanes", [2, 8, 32])
def test_dpc_prefilter(gpu_pkg, orc, D, lanes):
    """dpcreg! with pairs on both sides of l₀ (fluid jittered by up to a
    quarter of the spacing, l₀ = 0.7 dx): the FP32 test must pass on every pair
    the FP64 one takes."""
    case = _case(gpu_pkg, D, (1, 0, 0))
    rng = np.random.default_rng(3)
    fl = case.ptype > 1
    case.x[:, fl] += rng.uniform(-0.2, 0.2, (D, int(fl.sum()))) * case.dx
    case.extra = dict(case.extra, dpc_l0=0.7 * case.dx, dpc_lambda=0.005, dpc_pmax=36000.0)
    v = well_conditioned_v(case)
    prob, ref = make_pair(gpu_pkg, orc, case, lanes, v=v)
    run_both(prob, ref, 6)
    assert np.abs(ref.get("buf2")).max() > 0
    check(orc, prob, ref, case, lanes, [(6, {})], v=v)


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("lanes", [2, 4, 32])
def test_sums_without_a_step(gpu_pkg, orc, D, lanes):
    """A call of no steps sums W and ∇W over the caller's points through the
    map, one of a step over the cell-order state."""
    case = _case(gpu_pkg, D, (1, 0, 0))
    prob, ref = make_pair(gpu_pkg, orc, case, lanes)
    for n in (0, 1):
        run_both(prob, ref, n)
        for f in ("sumW", "sumgW"):
            got, want = prob.field(f), ref.get(f)
            got = np.stack([t.cpu().numpy() for t in got]) if isinstance(got, tuple) else got.cpu().numpy()
            # eight roundings per term of up to 200 terms against ∑|terms| <= 4x the largest sum
            assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max(), f


@pytest.mark.parametrize("D", [2, 3])
def test_rows_by_a_thread_per_point(gpu_pkg, orc, D):
    """Sets past 32,768 particles search their rows with a thread per point:
    on serial rows, whose sums follow the rows' order, two calls are the
    oracle's to the bit."""
    if D == 2:
        case = gpu_pkg.workloads.dam_break_2d(dx=0.0078)
    else:
        case = gpu_pkg.workloads.dam_break_3d(dx=0.042, fluid=(1.0, 1.2, 0.7), tank=(2.4, 1.6, 1.2), full_physics=False)
    assert 32768 <= case.N <= 65536
    rng = np.random.default_rng(2)
    fl = case.ptype > 1
    case.x = case.x.copy()
    case.x[:, fl] += rng.uniform(-0.2, 0.2, (D, int(fl.sum()))) * case.dx
    prob, ref = make_pair(gpu_pkg, orc, case, 1)
    for _ in range(2):
        run_both(prob, ref, 1)
    check(orc, prob, ref, case, 1, [(1, {}), (1, {})])


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("factor", [1.02, 1.1, 1.4])
@pytest.mark.parametrize("s", [0.0, 0.05])
def test_pairs_past_the_reach(gpu_pkg, orc, D, factor, s):
    """Lists with a skin hold pairs past H, which pass A tells apart from 3% on
    (more pairs than its blocks have threads): over steps that keep the list
    and steps that bring pairs into reach."""
    if D == 2:
        case = gpu_pkg.workloads.dam_break_2d(dx=0.0156, layer_ptype=(1, 0, -1), dist_factor=factor)
    else:
        case = gpu_pkg.workloads.dam_break_3d(dx=0.05, fluid=(0.5, 0.6, 0.4), tank=(1.0, 0.8, 0.6),
                                              layer_ptype=(1, 0, -1), full_physics=False)
        case.dist = factor * case.H
        case.cellsize = (case.dist,) * 3
    case.s = s
    case.extra = dict(nu=0.2, xsph_eps=0.5, cspmn=3)
    # walls too: lattice walls of both signs hold pairs at exactly r₀, where the
    # root's last bit decides fbmolforce!
    rng = np.random.default_rng(17)
    case.x = case.x + rng.uniform(-0.2, 0.2, case.x.shape) * case.dx
    case.rho = case.rho + rng.uniform(0.0, 2.0, case.rho.size)
    v = well_conditioned_v(case)
    prob, ref = make_pair(gpu_pkg, orc, case, 4, v=v)
    assert prob.system.pairsn > 152 * 768
    for _ in range(2):
        run_both(prob, ref, 3)
    check(orc, prob, ref, case, 4, [(3, {}), (3, {})], v=v)
