"""fbmolforce! at exactly r₀: lattice walls hold pairs at two spacings, where the
last bit of the separation decides whether a pair has a force.  Split rows
decide as the reference does (0.0078, 0.013 and 0.0156 are spacings at which an
approximate root decides some of them the other way)."""
import numpy as np
import pytest

from test_sph_gpu import check, make_pair, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,dx", [(2, 0.0078), (2, 0.013), (2, 0.0156), (3, 0.052)])
@pytest.mark.parametrize("layers", [(1, 0, 0), (1, 0, -1)])
def test_pairs_at_the_cut(gpu_pkg, orc, D, dx, layers):
    if D == 2:
        case = gpu_pkg.workloads.dam_break_2d(dx=dx, fluid=(0.5, 0.6), tank=(1.0, 0.8), layer_ptype=layers)
    else:
        case = gpu_pkg.workloads.dam_break_3d(dx=dx, fluid=(0.3, 0.4, 0.3), tank=(0.6, 0.6, 0.4), layer_ptype=layers,
                                              full_physics=False)
    rng = np.random.default_rng(9)
    case.rho = case.rho + rng.uniform(0.0, 2.0, case.rho.size)
    for lanes in (2, 4, 32):
        prob, ref = make_pair(gpu_pkg, orc, case, lanes)
        run_both(prob, ref, 1)
        check(orc, prob, ref, case, lanes, [(1, {})])
