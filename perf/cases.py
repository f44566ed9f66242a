"""The framework's work as its users call it, as a list of cases that can be timed and checked.

Every case goes through the public Python API: the cell list (GPUCellList, update!, partialupdate!), the
FP64 solver (SPHProblem, stepsolve!), the exported kernel functions on a pair list, and the batched FP32
ensemble.  `exact` is a plain torch statement of the same equations in 64 bits.
"""
import math

import numpy as np
import torch

import __graft_entry__

g = __graft_entry__.load_package()


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # An interactive or coupled host calls stepsolve!(prob, 1) and looks at the state after every
        # step: the smallest call, launches and round trips count (2-D dam break, 6.5 k particles).
        {"name": "step2d-single", "kind": "step", "D": 2, "fluid": 5000, "aspect": 2.0, "dx": 0.02, "steps": 1,
         "full": False, "skin": 1.0, "adaptive": False},
        # The reference's headline run: the 2-D dam break, plain FP64, cell list rebuilt every step, in
        # batches of 15 steps (one CSPM period).
        {"name": "step2d-batch", "kind": "step", "D": 2, "fluid": 5000, "aspect": 2.0, "dx": 0.02, "steps": 15,
         "full": False, "skin": 1.0, "adaptive": False},
        # A fine 2-D tank with every physics option of the solver, a pair list with a skin (dist = 1.1 H)
        # that is kept over several steps, and Δt stepping; an odd particle count.
        {"name": "step2d-full-skin", "kind": "step", "D": 2, "fluid": 60001, "aspect": 1.3, "dx": 0.005, "steps": 10,
         "full": True, "skin": 1.1, "adaptive": True},
        # A small 3-D tank, plain physics, list rebuilt every step: most particles are walls.
        {"name": "step3d-plain", "kind": "step", "D": 3, "fluid": 20000, "aspect": 1.7, "dx": 0.02, "steps": 5,
         "full": False, "skin": 1.0, "adaptive": False},
        # The 3-D dam break of the examples with viscosity, surface tension, DPC and XSPH in FP64
        # (390 k particles): the largest FP64 solve that runs interactively.
        {"name": "step3d-full", "kind": "step", "D": 3, "fluid": 125000, "aspect": 2.0, "dx": 0.02, "steps": 3,
         "full": True, "skin": 1.0, "adaptive": False},
        # The cell list alone at the size the reference publishes: update! of 200 k uniform 2-D points,
        # about 80 pairs a point.
        {"name": "list2d-update", "kind": "list", "D": 2, "points": 200000, "per_point": 80.0, "op": "update"},
        # The cell list at scale: update! of 4 M uniform 3-D points, few pairs a point.
        {"name": "list3d-update", "kind": "list", "D": 3, "points": 4000000, "per_point": 4.3, "op": "update"},
        # partialupdate! between full rebuilds: points moved, cells kept; a ragged 3-D set.
        {"name": "list3d-partial", "kind": "list", "D": 3, "points": 333331, "per_point": 45.0, "op": "partial"},
        # A host that composes its own step from the exported kernel functions, at the size at which the
        # reference times them.
        {"name": "kernels2d", "kind": "kernels", "D": 2, "fluid": 5000, "aspect": 2.0, "dx": 0.02},
        # The same composition for a 3-D tank at scale (millions of pairs).
        {"name": "kernels3d", "kind": "kernels", "D": 3, "fluid": 50000, "aspect": 1.0, "dx": 0.01},
        # A parameter study: 20 independent 2-D dam breaks of different sizes, α and δ advanced
        # together in FP32, 60 steps a call, every instance's fields read back.
        {"name": "ens2d-batch", "kind": "ens", "D": 2, "instances": 20, "lo": 3000, "hi": 100000, "steps": 60,
         "full": False},
        # One 3-D solve with full physics on the FP32 engine, as the serving loop runs it.
        {"name": "ens3d-full", "kind": "ens", "D": 3, "instances": 1, "lo": 125000, "hi": 125000, "steps": 30,
         "full": True},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "list", "list", "kernels", "ens", "ens"))
    D = rng.choice((2, 3))
    if kind == "step":
        fluid = int(_log(rng, 600, 80000)) if D == 2 else int(_log(rng, 1500, 60000))
        return {"kind": kind, "D": D, "fluid": fluid, "aspect": round(rng.uniform(0.5, 3.0), 3),
                "dx": round(rng.uniform(0.005, 0.02), 4), "steps": rng.randint(1, 20 if D == 2 else 3),
                "full": rng.random() < 0.5, "skin": rng.choice((1.0, 1.0, 1.1)), "adaptive": rng.random() < 0.3}
    if kind == "list":
        per = round(_log(rng, 3.0, 90.0), 2)
        top = min(4000000, 1.5e7 / per)
        return {"kind": kind, "D": D, "points": int(_log(rng, 2000, top)), "per_point": per,
                "op": rng.choice(("update", "partial"))}
    if kind == "kernels":
        fluid = int(_log(rng, 600, 80000)) if D == 2 else int(_log(rng, 1500, 40000))
        return {"kind": kind, "D": D, "fluid": fluid, "aspect": round(rng.uniform(0.5, 3.0), 3),
                "dx": round(rng.uniform(0.005, 0.02), 4)}
    hi = int(_log(rng, 3000, 90000 if D == 2 else 40000))
    return {"kind": kind, "D": D, "instances": rng.randint(1, 16 if D == 2 else 3), "lo": max(1500, hi // 8), "hi": hi,
            "steps": rng.randint(10, 40 if D == 2 else 15), "full": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _tank(D, fluid, aspect, dx):
    make = g.workloads.sized_dam_break_2d if D == 2 else g.workloads.sized_dam_break_3d
    return make(int(fluid), float(aspect), float(dx))


def _flow(c, seed, full):
    """A dam break some way into its run: fluid off the lattice and out of the walls' repulsion (2 dx), hydrostatic
    density, a velocity field."""
    rng = np.random.Generator(np.random.PCG64([int(seed), 71]))
    fl = c.ptype > 1
    nf = int(fl.sum())
    x = c.x.copy()
    x[:, fl] += rng.uniform(-0.1, 0.1, (c.D, nf)) * c.dx + 1.1 * c.dx
    depth = np.maximum(x[1][fl].max() - x[1], 0.0)
    b = c.c0 * c.c0 * c.rho0 / c.gamma
    c.x = x
    c.rho = c.rho0 * (1.0 + c.rho0 * c.g * depth / b) ** (1.0 / c.gamma) + rng.uniform(0.0, 0.3, c.N)
    v = np.zeros_like(x)
    v[:, fl] = rng.normal(0.0, 0.2, (c.D, nf))
    if full:
        c.s = 0.05
        c.extra = dict(nu=0.2, dpc_l0=0.5 * c.dx, dpc_lambda=0.005, dpc_pmax=36000.0, xsph_eps=0.5)
    return v


def _problem(case, seed):
    c = _tank(case["D"], case["fluid"], case["aspect"], case["dx"])
    v = _flow(c, seed, case.get("full", False))
    c.dist = case.get("skin", 1.0) * c.H
    c.cellsize = (c.dist,) * c.D
    return c, v


def _ens_cases(case, seed):
    out = []
    for i in range(case["instances"]):
        # sizes belong to the case, the state to the seed
        size = np.random.Generator(np.random.PCG64([case["instances"], case["hi"], i]))
        n = math.exp(size.uniform(math.log(case["lo"]), math.log(case["hi"] + 1)))
        c = _tank(case["D"], n, size.uniform(0.5, 3.0) if case["instances"] > 1 else 2.0,
                  size.uniform(0.005, 0.02) if case["instances"] > 1 else 0.02)
        c.alpha, c.delta = float(size.uniform(0.005, 0.05)), float(size.uniform(0.05, 0.2))
        v = _flow(c, int(seed) * 64 + i, case["full"])
        out.append((c, v))
    return out


def _radius(D, n, per_point):
    """Cut-off at which n uniform points in the unit box have per_point pairs each."""
    ball = math.pi if D == 2 else 4.0 * math.pi / 3.0
    return (2.0 * per_point / (n * ball)) ** (1.0 / D)


def _capacity(D, n, r):
    """Room for the pairs of n uniform points in the unit box: the expected count and a ninth more."""
    p = (math.pi * r**2 - 8.0 / 3.0 * r**3 + 0.5 * r**4 if D == 2 else
         4.0 / 3.0 * math.pi * r**3 - 1.5 * math.pi * r**4 + 1.6 * r**5 - r**6 / 6.0)
    return int(1.11 * 0.5 * n * (n - 1) * p) + 1


def prepare(case, seed):
    if case["kind"] == "list":
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        x = torch.rand((case["D"], case["points"]), generator=gen, device="cuda", dtype=torch.float64)
        r = _radius(case["D"], case["points"], case["per_point"])
        D = case["D"]
        system = g.GPUCellList(tuple(x), (r,) * D, r, MIN=(0.0,) * D, MAX=(1.0,) * D,
                               mpairs=_capacity(D, case["points"], r))
        if case["op"] == "partial":
            for p in system.points:
                p += 0.02 * r * (torch.rand(p.shape, generator=gen, device="cuda", dtype=torch.float64) - 0.5)
        return {"case": case, "system": system}
    if case["kind"] == "ens":
        ens = g.Ensemble(case["D"])
        slots = []
        for c, v in _ens_cases(case, seed):
            spec = g.spec_from_case(c)
            spec.v = v
            slots.append(ens.add(spec))
        return {"case": case, "ens": ens, "slots": slots}
    c, v = _problem(case, seed)
    if case["kind"] == "kernels":
        # room for the pairs from the lattice's own list; the arrays per pair are as long as the list
        lattice = _tank(case["D"], case["fluid"], case["aspect"], case["dx"])
        room = int(1.1 * g.GPUCellList(tuple(lattice.x), c.cellsize, c.dist).pairsn)
        system = g.GPUCellList(tuple(c.x), c.cellsize, c.dist, mpairs=room)
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        f64 = lambda n: torch.zeros(n, dtype=torch.float64, device="cuda")  # noqa: E731
        P, N = len(g.neighborlist(system)), c.N
        return {"case": case, "c": c, "system": system, "pairs": g.neighborlist(system),
                "kernel": g.WendlandC2(dim=c.D), "rho": dev(c.rho), "v": tuple(dev(a) for a in v),
                "ptype": dev(c.ptype), "W": f64(P), "gW": tuple(f64(P) for _ in range(c.D)), "sumW": f64(N),
                "drho": f64(N), "P": f64(N), "a": tuple(f64(N) for _ in range(c.D)),
                "xs": tuple(f64(N) for _ in range(c.D))}
    system = g.GPUCellList(tuple(c.x), c.cellsize, c.dist)
    prob = g.SPHProblem(system, c.dx, c.h, c.H, g.WendlandC2(dim=c.D), c.rho, c.ptype, c.rho0, c.m0, c.dt, c.alpha,
                        c.c0, c.gamma, c.delta, c.CFL, v=tuple(v), g=c.g, s=c.s)
    for k, val in c.extra.items():
        setattr(prob, k, val)
    return {"case": case, "system": system, "prob": prob}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        prob = state["prob"]
        prob.stepsolve(case["steps"], timestepping=case["adaptive"])
        return {"x": g.get_points(prob), "v": g.get_velocity(prob), "rho": g.get_density(prob),
                "P": g.get_pressure(prob), "a": g.get_acceleration(prob)}
    if kind == "list":
        system = state["system"]
        if case["op"] == "update":
            g.update(system)
        else:
            g.partialupdate(system)
        return {"pairs": g.neighborlist(system), "cellpnum": system.cellpnum}
    if kind == "ens":
        ens = state["ens"]
        ens.step(case["steps"])
        # v and ρ - ρ₀ are held in 32 bits, x in 64
        return [{"x": ens.get(s, "x"), "v": ens.get(s, "v").astype(np.float32),
                 "drho": ens.get(s, "drho").astype(np.float32)} for s in state["slots"]]
    k, c = g.kernels, state["c"]
    pairs, x, v, rho, pt = state["pairs"], state["system"].points, state["v"], state["rho"], state["ptype"]
    W, gW, a, xs, kern = state["W"], state["gW"], state["a"], state["xs"], state["kernel"]
    k.sphW(W, pairs, x, 1.0 / c.H, kern)
    k.sphgradW(gW, pairs, x, 1.0 / c.H, kern)
    state["sumW"].zero_()
    k.sphsumW(state["sumW"], pairs, x, kern, 1.0 / c.H, pt)
    k.drhodtDDT(state["drho"], pairs, gW, rho, v, x, c.h, c.m0, c.rho0, c.c0, c.gamma, c.g, c.delta, pt)
    k.pressure(state["P"], rho, c.c0, c.gamma, c.rho0, pt)
    for t in a + xs:
        t.zero_()
    k.dvdt(a, gW, state["P"], pairs, c.m0, rho, pt)
    k.dvdt_av(a, gW, pairs, x, c.h, rho, c.alpha, v, c.c0, c.m0, pt)
    k.dvdt_visc(a, gW, v, rho, x, pairs, c.h, c.m0, 0.2, pt)
    k.dvdtpF(a, pairs, x, 0.05, c.h, c.m0, pt)
    k.fbmolforce(a, pairs, x, 0.4, 2.0 * c.dx, pt)
    k.dvdt_addgrav(a, c.g)
    k.xsphcorr(xs, pairs, W, rho, v, c.m0, 0.5, pt)
    return {"W": W, "gW": gW, "sumW": state["sumW"], "drho": state["drho"], "P": state["P"], "a": a, "xs": xs}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _counts(case):
    """Particles and pairs of a tank, from the lattice: a particle's H-ball holds about πH²/dx² points in
    2-D and 4πH³/3dx³ in 3-D; walls three layers deep see about half of that."""
    out = []
    if case["kind"] == "ens":
        sizes = []
        for i in range(case["instances"]):
            size = np.random.Generator(np.random.PCG64([case["instances"], case["hi"], i]))
            n = math.exp(size.uniform(math.log(case["lo"]), math.log(case["hi"] + 1)))
            sizes.append((n, size.uniform(0.5, 3.0) if case["instances"] > 1 else 2.0))
    else:
        sizes = [(case["fluid"], case["aspect"])]
    for n, asp in sizes:
        if case["D"] == 2:
            w = math.sqrt(n / asp)
            walls = 3.0 * (4.0 * w + 2.0 * 1.5 * asp * w)
            per = math.pi * (2 * 1.2 * math.sqrt(2.0)) ** 2 / 2.0
        else:
            w = (2.0 * n / asp) ** (1.0 / 3.0)
            walls = 3.0 * (4.0 * w * w + 2.0 * 4.0 * w * 1.5 * asp * w + 2.0 * w * 1.5 * asp * w)
            per = 4.0 * math.pi / 3.0 * (2.0 * math.sqrt(3.0)) ** 3 / 2.0
        out.append((n + walls, n * per + walls * per * 0.4))
    return sum(a for a, _ in out), sum(b for _, b in out)


def work(case):
    D = case["D"]
    if case["kind"] == "list":
        n, pairs = case["points"], case["points"] * case["per_point"]
        # coordinates in, the pair list out; a distance test per pair
        return {"bytes": 8 * D * n + 8 * pairs, "flops": 3 * D * pairs}
    n, pairs = _counts(case)
    # both stages of a step: kernel, continuity with diffusion, momentum with artificial viscosity (about
    # 120 operations a pair in 2-D, 150 in 3-D), 60 more with viscosity, surface tension, DPC and XSPH
    per_pair = 2 * (120 if D == 2 else 150) + (60 if case.get("full") else 0)
    if case["kind"] == "kernels":
        # state in and sums out once, the pair list in and W and ∇W out once
        return {"bytes": n * (8 * (5 * D + 4) + 4) + pairs * (8 + 8 + 8 * D), "flops": pairs * (per_pair // 2 + 60)}
    if case["kind"] == "ens":
        # positions in 64 bits, v and ρ in 32, read and written once; the fields out as doubles
        return {"bytes": n * (2 * (8 * D + 4 * D + 4) + 8 * (2 * D + 1)), "flops": case["steps"] * pairs * per_pair}
    # state in and out once a call, P and a out, and the refreshed pair list out
    return {"bytes": n * (8 * 2 * (2 * D + 1) + 8 * (D + 1) + 4) + 8 * pairs, "flops": case["steps"] * pairs * per_pair}


# ---------------------------------------------------------------------------
# the same equations in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pairs(x, r):
    """Index pairs (i, j), i before j in cell order, with |xi - xj| < r."""
    D, n = x.shape
    cell = torch.floor((x - x.min(1, keepdim=True).values) / r).to(torch.int64) + 1
    dims = cell.max(1).values + 2
    key = cell[0] + dims[0] * (cell[1] + (dims[1] * cell[2] if D == 3 else 0))
    order = torch.argsort(key)
    skey = key[order].contiguous()
    xs = x[:, order]
    idx = torch.arange(n, device=x.device)
    I, J = [], []
    for dz in ((-1, 0, 1) if D == 3 else (0,)):
        for dy in (-1, 0, 1):
            row = skey + dims[0] * (dy + (dims[1] * dz if D == 3 else 0))
            lo, hi = torch.searchsorted(skey, row - 1), torch.searchsorted(skey, row + 1, right=True)
            lo = torch.maximum(lo, idx + 1)
            cnt = (hi - lo).clamp(min=0)
            if int(cnt.sum()) == 0:
                continue
            i = torch.repeat_interleave(idx, cnt)
            j = torch.arange(i.numel(), device=x.device) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt - lo, cnt)
            near = ((xs[:, i] - xs[:, j]) ** 2).sum(0) < r * r
            I.append(order[i[near]])
            J.append(order[j[near]])
    return torch.cat(I), torch.cat(J)


def _add(n, i, j, fi, fj):
    if fi.dim() == 1:
        return torch.zeros(n, dtype=fi.dtype, device=fi.device).index_add_(0, i, fi).index_add_(0, j, fj)
    return torch.stack([_add(n, i, j, p, q) for p, q in zip(fi, fj)])


def _norms(D, H):
    s = 7.0 / math.pi if D == 2 else 21.0 / (2.0 * math.pi)
    return s / H ** D, s / H ** (D + 1)


def _kernel(dx, H):
    """W and ∇W of WendlandC2 at the separations dx."""
    nw, ndw = _norms(dx.shape[0], H)
    r = (dx * dx).sum(0).sqrt()
    u = r / H
    t = (1.0 - u).clamp(min=0.0)
    return (1.0 + 4.0 * u) * t ** 4 * nw, dx * (-20.0 * u * t ** 3 * ndw / r), r


def _pow7(x):
    """The solver's x^(1/7): an integer guess and two Halley steps (its bias is part of the δ-SPH term)."""
    t = (0x36cd000000000000 + x.view(torch.int64) // 7).view(torch.float64)
    for _ in range(2):
        q = x / t ** 4
        t = t - t * (t ** 3 - q) / (4.0 * t ** 3 + 3.0 * q)
    return t


def _eos(rho, pt, c):
    p = c.c0 * c.c0 * c.rho0 / c.gamma * ((rho / c.rho0) ** c.gamma - 1.0)
    return torch.where((pt <= 1) & (rho < c.rho0), torch.zeros_like(p), p)


def _ddt(c, i, j, dx, dv, gw, rho, pt):
    """∂ρ/∂t with δ-SPH diffusion: both sides' pair values."""
    both = ((pt[i] > 0) & (pt[j] > 0)).to(dx.dtype)
    inv = 1.0 / ((dx * dx).sum(0) + (0.1 * c.h) ** 2)
    kh = 2.0 * c.h * c.delta * c.c0
    gz = c.rho0 * c.g * c.gamma / (c.c0 * c.c0 * c.rho0)
    dot, base = -(dx * gw).sum(0) * c.m0, c.m0 * (dv * gw).sum(0)
    dr = rho[j] - rho[i]
    si = kh * (dr - (c.rho0 * _pow7(1.0 + gz * dx[1]) - c.rho0)) * inv * dot / rho[j]
    sj = kh * (-dr - (c.rho0 * _pow7(1.0 - gz * dx[1]) - c.rho0)) * inv * dot / rho[i]
    return both * (base + si * (pt[i] > 1)), both * (base + sj * (pt[j] > 1))


def _momentum(c, i, j, dx, dv, gw, rho, P, pt, nu, s):
    """∂v/∂t of i from pressure, artificial and laminar viscosity and surface tension (j takes the negative)."""
    f = torch.where(pt[i] * pt[j] > 0, -c.m0 * (P[i] + P[j]) / (rho[i] * rho[j]), 0.0) * gw
    both = ((pt[i] > 0) & (pt[j] > 0)).to(dx.dtype)
    r2 = (dx * dx).sum(0)
    inv = both / (r2 + (0.1 * c.h) ** 2)
    cond = (dv * dx).sum(0)
    rs = rho[i] + rho[j]
    f = f + torch.where(cond < 0.0, 2.0 * c.alpha * c.c0 * c.h * c.m0 * cond * inv / rs, 0.0) * gw
    if nu > 0:
        f = f + 4.0 * nu * c.m0 * (dx * gw).sum(0) * inv / rs * dv
    if s > 0:
        r = r2.sqrt()
        q = s * torch.cos(1.5 * math.pi * r / (2.0 * c.h)) / (r + 0.1 * c.h) / c.m0
        f = f + both * torch.where(r < 2.0 * c.h, q, 0.0) * dx
    return f


def _wall(dx, i, j, pt, d, r0):
    r2 = (dx * dx).sum(0)
    r, e = r2.sqrt(), 0.01 * r0 * r0
    q = r0 / (r + e)
    on = ((pt[i] > 0) != (pt[j] > 0)) & (r < r0)
    return torch.where(on, d * (q ** 12 - q ** 4) / (r2 + e), 0.0) * dx


def _dpc(c, i, j, x, v, rho, P, pt, dt, ex):
    l0, nw = ex["dpc_l0"], _norms(x.shape[0], ex["dpc_l0"])[0]
    dx, dv = x[:, i] - x[:, j], v[:, i] - v[:, j]
    r2 = (dx * dx).sum(0)
    u = r2.sqrt() / l0
    w = lambda q: (1.0 + 4.0 * q) * (1.0 - q).clamp(min=0.0) ** 4 * nw  # noqa: E731
    chi = (w(u) / (1.5 * w(torch.zeros(1, dtype=u.dtype, device=u.device)) / 8.0)).sqrt()
    nx = _norms(x.shape[0], 1.0)[0]
    lo, hi = 0.0, 1.0  # W(u; H = 1) = 1
    for _ in range(200):
        m = 0.5 * (lo + hi)
        lo, hi = (m, hi) if (1.0 + 4.0 * m) * (1.0 - m) ** 4 * nx > 1.0 else (lo, m)
    k = torch.where(u < lo, torch.ones_like(chi), chi)
    pb = chi * (ex["dpc_lambda"] * (P[i] + P[j]).abs()).clamp(max=ex["dpc_lambda"] * ex["dpc_pmax"]).clamp(min=1.0)
    vr = (dv * dx).sum(0)
    e = r2 + (0.1 * l0) ** 2
    f = torch.where(vr < 0.0, -k * vr / e, 2.0 * dt * pb / ((rho[i] + rho[j]) * e)) * dx
    return torch.where((pt[i] > 0) & (pt[j] > 0) & (u < 1.0), f, torch.zeros_like(f))


def _solve(c, v0, steps, adaptive, skin=1.0):
    """`steps` steps of the symplectic scheme from (c.x, v0, c.rho): x, v, ρ, P, a.  A list with a skin keeps the
    pairs beyond H in the step (their kernel is zero), one without drops them at each step's start."""
    dev = _dev()
    f = lambda a: torch.as_tensor(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    x, v, rho, pt = f(c.x), f(v0), f(c.rho), f(c.ptype)
    D, n = x.shape
    ex, s = c.extra, c.s
    nu = ex.get("nu", 0.0)
    # one list for the call: wider than H by more than the particles move
    I, J = _pairs(x, skin * c.H + 2.0 * c.dx * min(1.0, 0.004 * steps + 0.02))
    dt = c.dt
    grav = torch.zeros((D, 1), dtype=x.dtype, device=dev)
    grav[1] = c.g
    fl = pt > 1
    xh, vh, rhoh = x.clone(), v.clone(), rho.clone()
    P = a = None
    for it in range(steps):
        dx = x[:, I] - x[:, J]
        near = (dx * dx).sum(0) < (skin * c.H) ** 2
        i, j, dx = I[near], J[near], dx[:, near]
        W, gw, _ = _kernel(dx, c.H)
        dv = v[:, i] - v[:, j]
        dr = _add(n, i, j, *_ddt(c, i, j, dx, dv, gw, rho, pt))
        fo = _momentum(c, i, j, dx, dv, gw, rho, _eos(rho, pt, c), pt, nu, s) + _wall(dx, i, j, pt, 0.4, 2.0 * c.dx)
        a = _add(n, i, j, fo, -fo) - grav
        rhoh = rhoh + dr * (0.5 * dt)
        vh = vh + torch.where(fl, a * (0.5 * dt), 0.0)
        xh = xh + vh * (0.5 * dt)
        P = _eos(rhoh, pt, c)
        dh, dvh = xh[:, i] - xh[:, j], vh[:, i] - vh[:, j]
        dr = _add(n, i, j, *_ddt(c, i, j, dh, dvh, gw, rhoh, pt))
        fo = _momentum(c, i, j, dh, dvh, gw, rhoh, P, pt, nu, s) + _wall(dx, i, j, pt, 0.4, 2.0 * c.dx)
        a = _add(n, i, j, fo, -fo) - grav
        e = -(dr / rhoh) * dt
        rho = rho * (2.0 - e) / (2.0 + e)
        rho = torch.where((rho < c.rho0) & (pt <= 1), torch.full_like(rho, c.rho0), rho)
        nv = v + torch.where(fl, a * dt, 0.0)
        x = x + 0.5 * (v + nv) * dt
        v = nv
        rhoh, vh, xh = rho, v, x
        if ex.get("dpc_l0", 0.0) > 0:
            P = _eos(rho, pt, c)
            fo = _dpc(c, i, j, x, v, rho, P, pt, dt, ex)
            q = torch.where(fl, _add(n, i, j, fo, -fo), 0.0)
            v, x = v + q, x + q * dt
        if ex.get("xsph_eps", 0.0) > 0:
            x = x + torch.where(fl, _xsph(c, i, j, W, rho, v, pt, ex["xsph_eps"]) * dt, 0.0)
        if (it + 1) % 15 == 0:
            real = ((pt[i] > 0) & (pt[j] > 0)).to(x.dtype) * W * c.m0
            s1, s2 = _add(n, i, j, real, real), _add(n, i, j, real / rho[j], real / rho[i])
            rho = torch.where(s2 > 0, s1 / s2, rho)
        if adaptive:
            am = float((a * a).sum(0).sqrt().max())
            vm = float((c.h * (v * x).sum(0) / ((x * x).sum(0) + (0.01 * c.h) ** 2)).abs().max())
            lim = (math.sqrt(2.220446049250313e-16), c.CFL * c.H / (3 * c.c0))
            dt = min(max(c.CFL * min(math.sqrt(c.h / (3.0 * am)), c.h / (c.c0 + vm)), lim[0]), lim[1])
    return x, v, rho, P, a


def _xsph(c, i, j, W, rho, v, pt, eps):
    q = torch.where((pt[i] > 1) & (pt[j] > 1), 2.0 * c.m0 * eps * W / (rho[i] + rho[j]), 0.0) * (v[:, j] - v[:, i])
    return _add(v.shape[1], i, j, q, -q)


def exact(case, seed):
    if case["kind"] == "list":
        return None  # whole numbers
    if case["kind"] == "ens":
        out = []
        for c, v in _ens_cases(case, seed):
            x, v, rho, _, _ = _solve(c, v, case["steps"], False)
            out.append({"x": x, "v": v, "drho": rho - c.rho0})
        return out
    c, v = _problem(case, seed)
    if case["kind"] == "step":
        x, v, rho, P, a = _solve(c, v, case["steps"], case["adaptive"], case["skin"])
        return {"x": tuple(x), "v": tuple(v), "rho": rho, "P": P, "a": tuple(a)}
    # the pair list's order belongs to the list: W and ∇W a pair are checked through the sums
    dev = _dev()
    f = lambda a: torch.as_tensor(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    x, v, rho, pt = f(c.x), f(v), f(c.rho), f(c.ptype)
    n = c.N
    i, j = _pairs(x, c.H)
    dx, dv = x[:, i] - x[:, j], v[:, i] - v[:, j]
    W, gw, _ = _kernel(dx, c.H)
    same = torch.where((pt[i] > 0) == (pt[j] > 0), W, torch.zeros_like(W))
    P = _eos(rho, pt, c)
    fo = _momentum(c, i, j, dx, dv, gw, rho, P, pt, 0.2, 0.05) + _wall(dx, i, j, pt, 0.4, 2.0 * c.dx)
    a = _add(n, i, j, fo, -fo)
    a[1] -= c.g
    return {"W": None, "gW": (None,) * c.D, "sumW": _add(n, i, j, same, same),
            "drho": _add(n, i, j, *_ddt(c, i, j, dx, dv, gw, rho, pt)), "P": P, "a": tuple(a),
            "xs": tuple(_xsph(c, i, j, W, rho, v, pt, 0.5))}
