// sph_step.cuh -- types and per-pair device helpers shared by the fused
// FP64 step kernels (sph_step.cu, compiled without FMA contraction so that
// the serial row order reproduces the CPU oracle bit for bit) and the
// pair-once split-row passes (sph_once.cu, compiled with contraction).
#pragma once
#include <math.h>
#include "celllist.cuh"
#include "pf7_series.cuh"

namespace gcsph {

static constexpr int STPB = 128;

constexpr int PF_COS_N = 13;
// pf_cos's coefficients times f
inline void pf_cos_coef(double f, double* C) {
  const double T[PF_COS_N] = {
      -0.9818965112591632,   0.31558602480454173, 1.2838905431807321,     -0.7879472662466167,   0.19547895338475096,
      -0.027475032586512103, 0.00251908751511393, -0.00016342789686839775, 7.918215700351492e-06, -2.9785382234404e-07,
      8.958338323810472e-09, -2.2072216601308446e-10, 4.5275475585621706e-12};
  for (int i = 0; i < PF_COS_N; ++i) C[i] = f * T[i];
}

struct StepConst {
  double h, eta2, m0, rho0, ginv, DDTkh, DDTgz, P0, alpha, c0, nu, g, s, Hinv, nW, nDW;
  double fb_d, fb_r0, fb_eta2;  // fbmolforce constants of the stage being run
  double fb_r2max;              // the largest r² whose (correctly rounded) root is below r₀; negative: none
  // pair-once products of the constants: m₀ d𝒲/r = dWr (1 - u)^3 (u / r = H⁻¹),
  // ∂v∂t_av!'s 2 α c₀ h and ∂v∂t_visc!'s 4 ν
  double dWr, avK, visc4;
  double dWg;                   // d𝒲/r = dWg (1 - u)^3 (∑∇W of a call)
  double twoh, pfc, hp1;        // 2h, 1.5*pi, 0.1h  (∂v∂tpF!)
  double pfk2;                  // 2 / (2h)² and s/m₀ times the cosine's coefficients (∂v∂tpF! of the pair-once pass)
  double pfc_s[PF_COS_N];
  double far_r2;                // (reach of the pair terms)² (1 + 1e-6) on lists that hold pairs well past it, else 0
  double dpc_l0inv, dpc_nW, dpc_whinv, dpc_pmin, dpc_pmax, dpc_lambda, dpc_kernlim, dpc_eta2;
  double dpc_r2cut;  // l0² (1 + 1e-6): past it u = √r² / l0 >= 1 whatever the rounding
  double xsph_c;                // 2*m0*eps
  double cfl, dt_eta2;          // Δt_stepping
  double tmin, tmax;
  int gamma, use_visc, use_pF, timestepping;
  int fold_end;    // pass B2's last block does k_step_end's work (no Δt_stepping in this call)
  int reset_max;   // the step's end clears the step's maxima for the next (captured calls: no memset node)
  double reb_thr;  // update! is due after a step whose max |cΔx| passes this (0.9 (dist - H))
  int dt_relative; // Δt_stepping's velocity term from pair-relative Δv·Δx instead of absolute v·x
  int count_reb;   // this step's decision counts toward the call's update! total
  int need_w;      // pass A stage 1 writes W: xsphcorr! or this step's cspmcorr! reads it
};

// device scalars of a running solve
struct Scal {
  double dt;
  double etime;
  unsigned long long maxcdx;  // bits of max |cΔx| of the current step
  unsigned long long amax;    // bits of max |a|
  unsigned long long vmax;    // bits of max |h v.x/(x.x+η²)|
  int ovf;                    // the neighbour CSR outgrew its buffers: this step's kernels skip
  unsigned bdone;             // blocks of pass B2 done this step (k_step_end's work in its last block)
  unsigned long long maxout;  // bits of the largest max |cΔx| of the call (stepsolve!'s second result)
  long long nreb;             // update! calls of the call (stepsolve!'s first result)
  int wild;                   // a velocity, density, 1/density or pressure was NaN or infinite in this call
};

template <int D>
struct SArr {
  const int64_t* rs;
  const int32_t* nbr;
  const int32_t* pt;
  const int32_t* orig;
  const int* ovf;  // set: the step's kernels skip (buffers outgrown, see rebuild)
  int* wild;       // Scal::wild
  double* x[3];
  double* v[3];
  double* rho;
  double* P1;
  double* xh[3];
  double* vh[3];
  double* rhoh;
  double* P2;
  double* ir;   // 1/ρ (pair-once stage 1)
  double* irh;  // 1/ρΔt½ (pair-once stage 2)
  double* We;
  double* gWe[3];  // ∇W per neighbour entry on serial rows, m₀∇W per pair of the flat list on split rows
  double* a[3];
  double* drho;
  double* cdx[3];
  double* buf2[3];
  double* Plast;
  double* xo[3];
  double* xho[3];
  double* vho[3];
  double* vo[3];
  double* rhoho;
  double* rhoo;
};

template <int D>
__device__ inline double dotD(const double* a, const double* b) {
  double s = a[0] * b[0];
#pragma unroll
  for (int d = 1; d < D; ++d) s = s + a[d] * b[d];
  return s;
}

// Julia min/max propagate NaN (fmin/fmax do not)
__device__ inline double jl_min(double a, double b) { return (a != a || b != b) ? (a + b) : fmin(a, b); }
__device__ inline double jl_max(double a, double b) { return (a != a || b != b) ? (a + b) : fmax(a, b); }

// the end of a step, one thread: etime += Δt (src/sphproblem.jl:331), the
// update! decision from max |cΔx| (:325-327), the call's largest max |cΔx|,
// and with Δt_stepping the next Δt from the step's maxima
__device__ inline void step_end_body(const StepConst& c, Scal* sc) {
  const double dt = sc->dt;
  sc->etime = sc->etime + dt;
  const double mc = __longlong_as_double((long long)sc->maxcdx);
  if (sc->maxcdx > sc->maxout) sc->maxout = sc->maxcdx;
  if (c.count_reb && mc > c.reb_thr) sc->nreb += 1;
  if (c.timestepping) {
    const double amax = __longlong_as_double((long long)sc->amax);
    const double vmax = __longlong_as_double((long long)sc->vmax);
    const double dt1 = sqrt(c.h / (3.0 * amax));
    const double dt2 = c.h / (c.c0 + vmax);
    double nd = c.cfl * jl_min(dt1, dt2);
    nd = jl_min(jl_max(nd, c.tmin), c.tmax);
    sc->dt = nd;
  }
  if (c.reset_max) {
    sc->maxcdx = 0ull;
    sc->amax = 0ull;
    sc->vmax = 0ull;
  }
}

// the exponent of x in its high word's place; HI_INF for infinities and NaN
__device__ __forceinline__ unsigned exponent(double x) {
  return (unsigned)((unsigned long long)__double_as_longlong(x) >> 32) & HI_INF;
}
__device__ __forceinline__ void note_wild(int* wild, unsigned top) {
  if (top == HI_INF) *wild = 1;
}

// ∂ρ∂tDDT! pair value seen from particle k (src/gpukernels_sph.jl:579-625)
template <int D>
__device__ inline double ddt_term(const StepConst& c, int ptk, int ptm, const double* dx, double r2, const double* gw,
                                  const double* dv, double rk, double rm) {
  if (!(ptk > 0 && ptm > 0)) return 0.0;
  double dot3 = -dotD<D>(dx, gw);
  double m0dot = c.m0 * dotD<D>(dv, gw);
  double s = m0dot;
  if (ptk > 1) {
    double drhopvp = c.rho0 * powfancy7th(1.0 + c.DDTgz * dx[1], c.ginv, c.gamma) - c.rho0;
    double visc_densi = c.DDTkh * ((rm - rk) - drhopvp) / (r2 + c.eta2);
    double delta = visc_densi * dot3 * c.m0 / rm;
    s += delta;
  }
  return s;
}

// all momentum terms of one pair seen from k; accumulators kept apart so the
// final sum follows the reference's kernel order (∂v∂t!, av, visc, grav, fb, pF)
template <int D>
struct Acc {
  double p[D], av[D], vi[D], fb[D], pf[D];
  __device__ void zero() {
#pragma unroll
    for (int d = 0; d < D; ++d) p[d] = av[d] = vi[d] = fb[d] = pf[d] = 0.0;
  }
};

template <int D>
__device__ inline void mom_terms(const StepConst& c, Acc<D>& A, int ptk, int ptm, const double* dx, double r2,
                                 const double* gw, const double* dv, double rk, double rm, double Pk, double Pm) {
  // ∂v∂t!, :755-772
  if (ptk * ptm > 0) {
    double Pfac = (Pk + Pm) / (rk * rm);
    double sc = -c.m0 * Pfac;
#pragma unroll
    for (int d = 0; d < D; ++d) A.p[d] += sc * gw[d];
  }
  if (ptk > 0 && ptm > 0) {
    // ∂v∂t_av!, :869-897
    double rhom = (rk + rm) * 0.5;
    double cond = dotD<D>(dv, dx);
    if (cond < 0.0) {
      double dmu = c.h * cond / (r2 + c.eta2);
      double dPi = (-c.alpha * c.c0 * dmu) / rhom;
      double sc = -dPi * c.m0;
#pragma unroll
      for (int d = 0; d < D; ++d) A.av[d] += sc * gw[d];
    }
    // ∂v∂t_visc!, :967-980
    if (c.use_visc) {
      double nuterm = 4.0 * c.nu * c.m0 * dotD<D>(dx, gw) / ((rk + rm) * (r2 + c.eta2));
#pragma unroll
      for (int d = 0; d < D; ++d) A.vi[d] += nuterm * dv[d];
    }
  }
}

// fbmolforce!, :1891-1901 (mask: exactly one side real)
template <int D>
__device__ inline void fb_term(const StepConst& c, Acc<D>& A, int ptk, int ptm, const double* dx, double r2) {
  if ((ptk > 0) == (ptm > 0)) return;
  double r = sqrt(r2);
  if (r < c.fb_r0) {
    double q = c.fb_r0 / (r + c.fb_eta2);
    double q2 = q * q, q4 = q2 * q2, q8 = q4 * q4, q12 = q8 * q4;
    double Fc = c.fb_d * (q12 - q4) / (r2 + c.fb_eta2);
#pragma unroll
    for (int d = 0; d < D; ++d) A.fb[d] += dx[d] * Fc;
  }
}

// ∂v∂tpF!, :1387-1397
template <int D>
__device__ inline void pf_term(const StepConst& c, Acc<D>& A, int ptk, int ptm, const double* dx, double r) {
  if (!(ptk > 0 && ptm > 0)) return;
  if (r < c.twoh) {
    double scos = c.s * gc_cos(c.pfc * r / c.twoh) / (r + c.hp1);
#pragma unroll
    for (int d = 0; d < D; ++d) A.pf[d] += scos * dx[d] / c.m0;
  }
}

// powfancy7th's step t - t(t³ - x/t⁴)/(4t³ + 3x/t⁴) in the equal form
// t - t(t⁷ - x)/(4t⁷ + 3x), with one division (the pair-once passes, outside
// the range of the series below)
__device__ inline double powfancy7th_1div(double x, double ginv, int gamma) {
  if (gamma != 7) return pow(x, ginv);
  const double ax = fabs(x);
  unsigned long long bits = (unsigned long long)__double_as_longlong(ax);
  bits = 0x36cd000000000000ULL + bits / 7ULL;
  double t = copysign(__longlong_as_double((long long)bits), x);
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const double t2 = t * t;
    const double t3 = t2 * t;
    const double t7 = t3 * (t2 * t2);
    t = t - (t * (t7 - x)) / (4.0 * t7 + 3.0 * x);
  }
  return t;
}

// a = ((((p + av) + visc) - g) + fb) + pF
template <int D>
__device__ inline void finish_acc(const StepConst& c, const Acc<D>& A, double* a) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    double v = A.p[d] + A.av[d];
    if (c.use_visc) v = v + A.vi[d];
    v = v - (d == 1 ? c.g : 0.0);
    v = v + A.fb[d];
    if (c.use_pF) v = v + A.pf[d];
    a[d] = v;
  }
}

// ---------------------------------------------------------------------------
// Sub-warp cooperation: L lanes (1, 2, 4, 8, 16 or 32) share one particle.
// Lane l walks row entries e0+l, e0+l+L, ...; the per-lane partial sums are
// combined across the lanes (sph_once.cu).  L = 1 is the serial row order -- the order the
// oracle's scatter over its canonically ordered pair list produces -- so it
// reproduces the oracle bit for bit; L > 1 re-associates the sums (within
// the FP64 contract) and fills the GPU when particles are few.
// ---------------------------------------------------------------------------
template <int L>
__device__ inline unsigned group_mask() {
  if constexpr (L == 32) {
    return 0xffffffffu;
  } else {
    const unsigned lanew = threadIdx.x & 31u;
    return ((1u << L) - 1u) << (lanew & ~(unsigned)(L - 1));
  }
}

// ---------------------------------------------------------------------------
// Pair-once stage passes (lanes > 1, the default).  The gather above
// evaluates every pair twice, once from each side; on GB300 the FP64 pipe is
// the bound, so here each pair is evaluated once.  Pass A: one thread per pair
// (k, m), k < m in cell order -- every thread has the same work, whatever the
// row lengths -- computes the pair and writes both sides' contributions into
// per-entry slots: slot e in k's row and slot mirror(e) in m's row.  Pass B:
// each particle sums its whole row (L lanes, fixed order -- deterministic, no
// atomics) and runs the predictor or the corrector.  Cost: one write + one
// read of a 32-byte slot per neighbour entry.  A slot is one DRAM and L2
// sector: the partner side's slots are scattered, and as separate arrays each
// of their 1 + D doubles touched a sector of its own.
// ---------------------------------------------------------------------------
struct __align__(32) PairOut {
  double rho, a[3];       // ∂ρ/∂t and ∂v/∂t (gravity not included); a[2] unused in 2-D
};
// a slot in one 32-byte access
__device__ __forceinline__ void put_slot(PairOut* p, double r, double a0, double a1, double a2) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(r), "d"(a0), "d"(a1), "d"(a2) : "memory");
}
// (the slots are read by a later launch than the one that wrote them)
__device__ __forceinline__ void get_slot(const PairOut* p, double* v) {
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}
struct PairBuf {
  PairOut* ce;            // per neighbour entry: the pair's contribution to that row's sums
  int4* pq;               // (k, m, e, mirror(e)) of every pair, k < m (mirror -1: stage 1 finds it)
  const int64_t* npair;   // number of pairs (device scalar)
};

// ---------------------------------------------------------------------------
// Pair-once arithmetic.  The FP64 pipe is the bound of pass A (2 FP64
// thread-instructions per cycle per SM on GB300), so its compares run on the
// integer pipe over the bit patterns, and its reciprocals and its root are
// polynomial corrections of the hardware's approximate reciprocal and
// reciprocal square root (rcp.approx / rsqrt.approx .f64, about 2^-20
// relative): one third-order step each, a result within a few ulp -- fewer FP64 instructions than the IEEE-rounded sequences, inside the
// FP64 contract this path is held to.
// ---------------------------------------------------------------------------
__device__ inline long long dbits(double x) { return __double_as_longlong(x); }
constexpr long long ONE_BITS = 0x3FF0000000000000LL;  // bits of 1.0
// x < 0.0 exactly as the FP compare (-0.0 and NaN are not), on the integer pipe
__device__ inline bool neg_int(double x) {
  return (unsigned long long)dbits(x) - 0x8000000000000001ull < 0x7FF0000000000000ull;
}

// 1/x, x normal: one third-order (Halley) step from the hardware's
// approximate reciprocal, y <- y (1 + e + e^2) with e = 1 - x y.  |e| is about
// 2^-20, so e^3 lies below the rounding; three FP64 instructions, where two
// Newton steps take four.
__device__ inline double rcp_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// the same where x may be 0 (or a denormal), infinite or NaN: there the
// approximation is the answer and the correction is NaN
__device__ inline double rcp_any(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0), r = fma(y, fma(e, e, e), y);
  return exponent(e) == HI_INF ? y : r;
}

// sqrt(x), x normal and positive: s = x y from the approximate reciprocal
// root y, then s (1 + e/2 + 3e^2/8) with e = 1 - s y (third order again): five
// FP64 instructions, where two Newton steps on the root and the product take
// eight.
__device__ inline double sqrt_nr(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double s = x * y;
  const double e = fma(-s, y, 1.0);
  return fma(s, e * fma(0.375, e, 0.5), s);
}

// cos(1.5π r/2h) of ∂v∂tpF! inside 2h, from r²: with s = 2 (r/2h)² - 1 it is
// cos(1.5π sqrt((1 + s)/2)), an entire function of s, and s covers [-1, 1];
// its Chebyshev series falls by about 100 a term there, and the series to the
// 12th degree (the next coefficient is 1.9e-17), in powers of s, is the
// polynomial (coefficients c_k = 2/M Σ f(cos θ_j) cos kθ_j over M = 64 points
// θ_j = π (j + 1/2)/M, c_0 halved, in 50 digits, then rounded).  k = 2/(2h)²; C
// holds the coefficients times the force's factor, in the launch's parameters,
// where they are operands of the FMAs.  13 FP64 instructions and no reduction,
// where a reduction by π/2 and a Taylor series took 16; the worst error against
// extended precision over 20 million separations in [0, 2h) is 8.2e-16, near 0.
__device__ inline double pf_cos(double r2, double k, const double* C) {
  const double s = fma(r2, k, -1.0);
  double p = C[PF_COS_N - 1];
#pragma unroll
  for (int i = PF_COS_N - 2; i >= 0; --i) p = fma(p, s, C[i]);
  return p;
}

// The exact Taylor series of powfancy7th's output (src/gpukernels_sph.jl:499-515,
// gen_pf7_series.py, bias included) in place of its two divisions: its terms past
// the constant, over d, the distance from the expansion point, by N coefficients of
// the side of 1 that d is on.
template <int N>
__device__ inline double pf7_poly(double d, const double* cu, const double* cl) {
  const bool up = dbits(d) >= 0;
  double r = up ? cu[N - 1] : cl[N - 1];
#pragma unroll
  for (int i = N - 2; i >= 0; --i) r = fma(r, d, up ? cu[i] : cl[i]);
  return r;
}
__device__ inline bool pf7_within(double d, double bound) {
  return (dbits(d) & 0x7FFFFFFFFFFFFFFFLL) <= dbits(bound);
}
// powfancy7th(1 + e) - 1, e taken as it is
__device__ inline double pf7m1_fast(double e, double ginv, int gamma) {
  static_assert(PF7_UP_N == PF7_LO_N, "series lengths");
  constexpr double A0U[PF7_UP_N] = PF7_UP_C, A0L[PF7_LO_N] = PF7_LO_C;
  static_assert(A0U[0] == A0L[0], "constant terms");
  if (gamma == 7 && pf7_within(e, PF7_EPS_MAX)) {
    const double cu[PF7_UP_N] = PF7_UP_C;
    const double cl[PF7_LO_N] = PF7_LO_C;
    const double r = pf7_within(e, PF7_EPS_SHORT) ? pf7_poly<PF7_SHORT_N - 1>(e, cu + 1, cl + 1)
                                                  : pf7_poly<PF7_UP_N - 1>(e, cu + 1, cl + 1);
    return fma(r, e, cu[0]);
  }
  return powfancy7th_1div(1.0 + e, ginv, gamma) - 1.0;
}
// powfancy7th(x) of the reference's rounded x = 1 + eps, and rounded once, as its
// t.  The step's passes take this: near rest ρ0 t - ρ0 is of the size of these
// roundings (without them a resting tank's largest ∂ρ/∂t, 1.9e-8, is 1.1e-12 of it
// off the oracle's).  The expansion point is a double at which t is one to
// a 500th of its last bit, so the polynomial's last step is the rounding.  (About
// 1, with the 1 in a constant that holds 1 + a₀ to 8e-18, 8% of the roots are an
// ulp off, and ∂ρ/∂t's error against extended precision is 1.4% larger in 2-D and
// 2.3% in 3-D; with the 1 added last, ten steps of 2-D full physics take 6149 us,
// about this point 6023; about it with the bounds asked of eps rather than of d, for
// the code's layout, 6134.)
__device__ inline double pf7_fast(double eps, double ginv, int gamma) {
  const double x = 1.0 + eps, d = x - (1.0 + PF7_ROOT_E);
  if (gamma == 7 && pf7_within(d, PF7_EPS_MAX)) {
    const double cu[PF7_UP_N - 1] = PF7_ROOT_UP_C;
    const double cl[PF7_LO_N - 1] = PF7_ROOT_LO_C;
    const double hu[PF7_SHORT_N - 1] = PF7_ROOT_HEAD_UP_C;
    const double hl[PF7_SHORT_N - 1] = PF7_ROOT_HEAD_LO_C;
    const double r = pf7_within(d, PF7_EPS_SHORT) ? pf7_poly<PF7_SHORT_N - 1>(d, hu, hl)
                                                  : pf7_poly<PF7_UP_N - 1>(d, cu, cl);
    return fma(r, d, PF7_ROOT_T);
  }
  return powfancy7th_1div(x, ginv, gamma);
}

// pair-once passes (sph_once.cu): pass A over the device-side pair count,
// one block per SM; pass B (row sums + predictor / corrector) with L lanes
// per particle, 32 particles per block
template <int D>
int launch_pairA(int stage, cudaStream_t st, const StepConst& c, const SArr<D>& S, const PairBuf& B, int64_t pairs_est);
// The next step's binning started by pass B2 (update! every step): each
// particle's cell key and arrival slot from its new position, and, in the
// last block, the cell starts (CellCore::sort with keys_ready goes on from
// there).  key == nullptr: none.
struct NextBin {
  int32_t* key;
  int32_t* slot;
  int32_t* count;      // zero on entry, zero again on exit
  int32_t* cellstart;
  Grid g;
};
// the caller's and the library's original-order arrays
template <int D>
struct StateIO {
  double* x[3];
  double* v[3];
  double* rho;
  const int32_t* pt;
  double* rhoh;
  double* vh[3];
  double* xh[3];
  double* cdx[3];
  double* a[3];
  double* drho;
  double* buf2[3];
  double* P;
};

// the FP32 copy (x - offset) of the particles' new positions that pass B2
// writes for dpcreg!'s prefilter; f[0] == nullptr: none
struct PosCopy {
  float* f[3];
  double off[3];
};
template <int D>
int launch_pairB(int stage, int L, int64_t N, cudaStream_t st, const StepConst& c, Scal* sc, const SArr<D>& S,
                 const PairBuf& B, const NextBin* nb = nullptr, const PosCopy* pc = nullptr);

// the gathers of a split-row step (L >= 2 lanes per particle)
template <int D>
int launch_dpc(int L, int64_t N, cudaStream_t st, const StepConst& c, const Scal* sc, const SArr<D>& S,
               const PosCopy& pc);
template <int D>
int launch_xsph(int L, int64_t N, cudaStream_t st, const StepConst& c, const Scal* sc, const SArr<D>& S);
template <int D>
int launch_cspm(int L, int64_t N, cudaStream_t st, const StepConst& c, const SArr<D>& S);
// ∑W and ∑∇W of a call.  X: the positions and pt the ptypes, by cell-order
// index (map null) or by map[cell-order index]; results go to orig's places.
// scatter: the cell-order state S goes to the original-order arrays O as well
// (k_scatter_state's work, without its launch).
struct PostSums {
  const double* x[3];
  const int32_t* pt;
  const int32_t* map;
  const int32_t* orig;
  double* sumW;
  double* sg[3];
};
template <int D>
int launch_sums_post(int L, int64_t N, cudaStream_t st, const StepConst& c, const int64_t* rs, const int32_t* nbr,
                     const PostSums& Q, const int* ovf, bool scatter, const StateIO<D>& O, const SArr<D>& S,
                     const PairBuf& B, int64_t pairs_est);

}  // namespace gcsph
