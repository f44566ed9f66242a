"""The summed pair terms of the exported kernels where their forms change: lists
long enough for the per-warp queues (over two resident grids of pairs) and just
under, ragged ends, unused rows, ptypes of every class, ε of the δ-SPH root
inside and outside its series, pairs on top of one another.  Against plain
numpy in 64 bits; a sum of n terms of the same size is bounded by n ulp of the
sum of their absolute values, here taken as 1e-12 of the largest sum."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("P,c0", [(1, 80.0), (33, 80.0), (100_003, 80.0), (1_900_001, 80.0), (1_900_001, 5.0)])
def test_terms_match_numpy(gpu_pkg, D, P, c0):
    K = gpu_pkg.kernels
    rng = np.random.default_rng(P + D)
    N = 5000
    h, H, dx, rho0, m0, g, delta, alpha, nu, s, eps = 0.05, 0.1, 0.04, 1000.0, 1.6, 9.81, 0.1, 0.02, 0.3, 0.05, 0.5
    x = 0.12 * rng.random((D, N))  # separations on both sides of every cut
    i = rng.integers(0, N, P)
    j = (i + rng.integers(1, N, P)) % N
    v = rng.normal(0, 0.3, (D, N))
    rho = rho0 * (1 + rng.uniform(-0.01, 0.01, N))
    Pr = rng.uniform(0, 1e4, N)
    pt = rng.choice(np.array([-1, 0, 1, 2, 2, 2], np.int32), N)
    pairs = np.stack([i, j], 1).astype(np.int32) + 1
    pairs[rng.random(P) < 0.05] = 0  # unused rows
    gW = rng.normal(0, 10.0, (D, P))
    W = rng.random(P)
    on = pairs[:, 0] > 0
    I, J = i[on], j[on]
    d, dv, gw, w = x[:, I] - x[:, J], v[:, I] - v[:, J], gW[:, on], W[on]
    r2 = (d * d).sum(0)
    r = np.sqrt(r2)
    pi, pj = pt[I], pt[J]
    both = (pi > 0) & (pj > 0)

    def add(fi, fj, mask):
        out = np.zeros(N)
        np.add.at(out, I[mask], fi[mask])
        np.add.at(out, J[mask], fj[mask])
        return out

    def vec(f, mask):
        return np.stack([add(f[q], -f[q], mask) for q in range(D)])

    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dvec = lambda a: tuple(dev(a[q]) for q in range(D))
    zero = lambda: tuple(torch.zeros(N, dtype=torch.float64, device="cuda") for _ in range(D))
    tp, tx, tv, tr, tpt, tgW, tP, tW = dev(pairs), dvec(x), dvec(v), dev(rho), dev(pt), dvec(gW), dev(Pr), dev(W)

    def same(got, want, what):
        got = np.stack([t.cpu().numpy() for t in got]) if isinstance(got, tuple) else got.cpu().numpy()
        err = np.abs(got - want).max()
        assert err <= 1e-12 * max(np.abs(want).max(), 1e-300), (what, err)

    # sph∑W!, sph∑∇W!
    nw = (7 / np.pi if D == 2 else 21 / (2 * np.pi)) / H**D
    u = r / H
    t = np.clip(1 - u, 0, None)
    real = (pi > 0) == (pj > 0)
    sW = torch.zeros(N, dtype=torch.float64, device="cuda")
    K.sphsumW(sW, tp, tx, None, 1 / H, tpt)
    wv = (1 + 4 * u) * t**4 * nw
    same(sW, add(wv, wv, real), "sumW")
    sg = zero()
    K.sphsumgradW(sg, tp, tx, None, 1 / H, tpt)
    same(sg, vec(d * (-20 * t**3 * nw / H**2), real), "sumgradW")
    # ∂ρ∂tDDT!
    gz, kh, inv = rho0 * g * 7 / (c0 * c0 * rho0), 2 * h * delta * c0, 1 / (r2 + 0.01 * h * h)

    def root(z):
        q = (0x36cd000000000000 + np.ascontiguousarray(z).view(np.uint64) // np.uint64(7)).view(np.float64)
        for _ in range(2):
            o = z / q**4
            q = q - q * (q**3 - o) / (4 * q**3 + 3 * o)
        return q
    dot, base = -(d * gw).sum(0) * m0, m0 * (dv * gw).sum(0)
    drr = rho[J] - rho[I]
    si = base + (pi > 1) * kh * (drr - (rho0 * root(1 + gz * d[1]) - rho0)) * inv * dot / rho[J]
    sj = base + (pj > 1) * kh * (-drr - (rho0 * root(1 - gz * d[1]) - rho0)) * inv * dot / rho[I]
    dr = torch.zeros(N, dtype=torch.float64, device="cuda")
    K.drhodtDDT(dr, tp, tgW, tr, tv, tx, h, m0, rho0, c0, 7, g, delta, tpt)
    same(dr, add(si, sj, both), "ddt")
    # the momentum terms
    a = zero()
    K.dvdt(a, tgW, tP, tp, m0, tr, tpt)
    same(a, vec(-m0 * (Pr[I] + Pr[J]) / (rho[I] * rho[J]) * gw, pi * pj > 0), "dvdt")
    a = zero()
    K.dvdt_av(a, tgW, tp, tx, h, tr, alpha, tv, c0, m0, tpt)
    cond = (dv * d).sum(0)
    same(a, vec(2 * alpha * c0 * h * m0 * cond * inv / (rho[I] + rho[J]) * gw, both & (cond < 0)), "av")
    a = zero()
    K.dvdt_visc(a, tgW, tv, tr, tx, tp, h, m0, nu, tpt)
    same(a, vec(4 * nu * m0 * (d * gw).sum(0) * inv / (rho[I] + rho[J]) * dv, both), "visc")
    a = zero()
    K.dvdtpF(a, tp, tx, s, h, m0, tpt)
    same(a, vec(s * np.cos(1.5 * np.pi * r / (2 * h)) / (r + 0.1 * h) / m0 * d, both & (r < 2 * h)), "pF")
    a = zero()
    K.fbmolforce(a, tp, tx, 0.4, 2 * dx, tpt)
    e = 0.01 * (2 * dx) ** 2
    q = 2 * dx / (r + e)
    same(a, vec(0.4 * (q**12 - q**4) / (r2 + e) * d, ((pi > 0) != (pj > 0)) & (r < 2 * dx)), "fb")
    a = zero()
    K.xsphcorr(a, tp, tW, tr, tv, m0, eps, tpt)
    same(a, vec(-dv * (2 * m0 * eps * w / (rho[I] + rho[J])), (pi > 1) & (pj > 1)), "xsph")


def test_coincident_points(gpu_pkg):
    """Two particles on top of one another: ∑∇W is the reference's 0/0, the
    other terms stay finite."""
    K = gpu_pkg.kernels
    f = lambda *q: torch.tensor(q, dtype=torch.float64, device="cuda")
    x, pt = (f(0.5, 0.5, 0.52), f(0.5, 0.5, 0.5)), torch.tensor([2, 2, 2], dtype=torch.int32, device="cuda")
    pairs = torch.tensor([[1, 2], [1, 3]], dtype=torch.int32, device="cuda")
    sW, sg, a = f(0, 0, 0), (f(0, 0, 0), f(0, 0, 0)), (f(0, 0, 0), f(0, 0, 0))
    K.sphsumW(sW, pairs, x, None, 10.0, pt)
    K.sphsumgradW(sg, pairs, x, None, 10.0, pt)
    K.dvdtpF(a, pairs, x, 0.05, 0.05, 1.0, pt)
    assert torch.isfinite(sW).all() and torch.isfinite(a[0]).all()
    assert torch.isnan(sg[0][:2]).all() and torch.isfinite(sg[0][2])
