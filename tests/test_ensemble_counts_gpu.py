"""An ensemble's stage passes take their constants from the launch's parameters
(one instance; up to 64) or from the table in memory (more): an instance's
results are bit-identical whichever it is, with each option that the constants
select and through instances that leave and join at the limits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "rho", "P", "ptype")


def _specs(pkg, D):
    w = pkg.workloads
    if D == 2:
        case = w.dam_break_2d(dx=0.05, fluid=(0.3, 0.4), tank=(0.6, 0.6))
    else:
        case = w.dam_break_3d(dx=0.06, fluid=(0.18, 0.3, 0.18), tank=(0.36, 0.48, 0.3), full_physics=False)
    plain = pkg.spec_from_case(case)
    visc = pkg.spec_from_case(case)
    visc.nu, visc.s, visc.gamma = 0.2, 0.05, 5
    full = pkg.spec_from_case(case)
    full.dpc_l0, full.dpc_lambda, full.dpc_pmax, full.xsph_eps, full.cspmn = 0.01, 0.005, 36000.0, 0.1, 4
    return plain, visc, full


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("count", [2, 64, 65])
@pytest.mark.parametrize("skin", [0.0, 0.1])
def test_results_do_not_depend_on_the_count(gpu_pkg, D, count, skin):
    specs = _specs(gpu_pkg, D)
    want = []
    for s in specs:
        one = gpu_pkg.Ensemble(D)
        one.set_skin(skin)
        slot = one.add(s)
        one.step(5)
        one.step(6)
        want.append({f: one.get(slot, f) for f in FIELDS})
        one.close()
    ens = gpu_pkg.Ensemble(D)
    ens.set_skin(skin)
    slots = [ens.add(specs[(k + count) % 3]) for k in range(count)]
    ens.step(5)
    ens.remove(slots[0])  # every other instance moves up ...
    late = ens.add(specs[0])  # ... and one joins behind them
    ens.step(6)
    for k in {1, count // 2, count - 1}:
        for f in FIELDS:
            assert np.array_equal(ens.get(slots[k], f), want[(k + count) % 3][f]), (k, f)
    assert ens.info(late)["steps"] == 6
    ens.close()
