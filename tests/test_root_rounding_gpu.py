"""∂ρ∂tDDT!'s root on split rows.  Near rest ρ₀ t - ρ₀ is of the size of t's last
bit, so t is to be the reference iteration's real value at the rounded 1 + ε,
rounded once.  20,000 isolated pairs at rest, whose ∂ρ/∂t is that term alone,
against the same in extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _root(x):
    """The iteration in extended precision (long double), x in doubles."""
    t = (np.int64(0x36CD000000000000) + x.view(np.int64) // 7).view(np.float64).astype(np.longdouble)
    for _ in range(2):
        q = x / t**4
        t = t - t * (t**3 - q) / (4 * t**3 + 3 * q)
    return t


@pytest.mark.parametrize("c0", [20.0, 60.0])
def test_the_root_is_rounded_once(gpu_pkg, c0):
    side, dx = 100, 0.01
    h = 1.2 * dx * np.sqrt(2.0)
    H = 2.0 * h
    rng = np.random.default_rng(21)
    gx, gy = np.meshgrid(np.arange(side) * 4.0 * H, np.arange(2 * side) * 4.0 * H, indexing="ij")
    first = np.stack([gx.ravel(), gy.ravel()])
    n = first.shape[1]
    r, phi = rng.uniform(0.3, 0.9, n) * H, rng.uniform(0.2, np.pi - 0.2, n)
    x = np.concatenate([first, first + r * np.stack([np.cos(phi), np.sin(phi)])], axis=1)
    N = 2 * n
    rho0, m0, delta, gamma, g = 1000.0, 1000.0 * dx * dx, 0.1, 7, 9.81
    c = gpu_pkg.GPUCellList(tuple(x), (H, H), H)
    assert c.pairsn == n
    prob = gpu_pkg.SPHProblem(c, dx, h, H, gpu_pkg.WendlandC2(dim=2), np.full(N, rho0), np.full(N, 2, np.int32), rho0,
                              m0, 1e-25, 0.0, c0, gamma, delta, 0.2, g=g)
    prob.set_lanes(2)
    prob.stepsolve(1)  # nothing moves: both stages see these positions
    got = prob.field("drhodt").cpu().numpy()

    L = np.longdouble
    for side_, sgn in ((slice(0, n), 1.0), (slice(n, N), -1.0)):
        d = sgn * (x[:, :n] - x[:, n:])
        gz = rho0 * g / ((c0 * c0 * rho0) * (1.0 / gamma))
        t = _root(1.0 + gz * d[1]).astype(np.float64)  # rounded once
        dp = (L(rho0) * t - L(rho0))
        dl = d.astype(L)
        r2 = (dl * dl).sum(0)
        u = np.sqrt(r2) / L(H)
        dw_r = -20 / L(H) * (1 - u) ** 3 * 7 / (L(np.pi) + L(1.2246467991473532e-16)) / L(H) ** 3
        want = 2 * L(h) * L(delta) * L(c0) * -dp / (r2 + (L(0.1) * L(h)) ** 2) * (-r2 * dw_r * L(m0)) / L(rho0)
        # t's neighbour is ρ₀ 2^-53 of dp away at least; everything else stays
        # within 64 roundings (7e-15) of the value
        ulp = np.abs(rho0 * 2.0**-53 / dp)
        assert ulp.min() > 4 * 64 * 2.0**-53
        off = np.abs(got[side_] / want - 1) > 0.5 * ulp
        # the series' last step is within 2^-53 of its |t - 1| < 2^-7 of the real
        # value: a rounding the other way at 2^-7 of the points at most
        assert off.mean() < 2.0**-7
