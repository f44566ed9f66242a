// sph_pairs.cu -- the reference's exported kernel functions as C-ABI calls.
//
// Each entry point takes the caller's pair list (1-based (i,j), rows with
// i == 0 skipped) and caller arrays in original particle order, and follows the
// reference kernel of the same name (src/gpukernels_sph.jl): one thread per
// pair, FP64 atomics into both particles.  These are the drop-in for users who
// call the kernels one by one; stepsolve! itself runs the fused gather path in
// sph_step.cu.
//
// What is written per pair or per particle (W, ∇W, P, the updates) keeps the
// reference's expressions and IEEE divisions and roots, bit for bit.  The
// terms that go into sums are bound by the FP64 pipe (80 to 87% busy, the
// atomics well behind), so they take the pair-once forms of the fused step:
// reciprocals, roots and the cosine by rcp_pair, sqrt_pair and pf_cos,
// powfancy7th by its series, dot products and products of constants fused.
// Measured with the queue below (one GB300, 10.5M pairs of a 3-D tank, 179k
// particles): ∂v∂tpF! 1577 -> 366 us, ∂ρ∂tDDT! 1403 -> 403, sph∑W! 499 -> 310,
// ∂v∂t_visc! 475 -> 281, fbmolforce! 449 -> 223, ∂v∂t_av! 425 -> 263, ∂v∂t! 231 -> 180,
// xsphcorr! 179 -> 151.
#include <math.h>
#include "sph_step.cuh"

namespace gcsph {

static constexpr int PTPB = 256;

struct V3 {
  const double* p[3];
};
struct W3 {
  double* p[3];
};

static int vec_in(int D, const double* const* src, V3* out, const char* name) {
  if (!src) return fail(GCSPH_EINVAL, "null %s", name);
  for (int d = 0; d < 3; ++d) out->p[d] = nullptr;
  for (int d = 0; d < D; ++d) {
    if (!src[d]) return fail(GCSPH_EINVAL, "null %s[%d]", name, d + 1);
    out->p[d] = src[d];
  }
  return GCSPH_OK;
}
static int vec_out(int D, double* const* src, W3* out, const char* name) {
  if (!src) return fail(GCSPH_EINVAL, "null %s", name);
  for (int d = 0; d < 3; ++d) out->p[d] = nullptr;
  for (int d = 0; d < D; ++d) {
    if (!src[d]) return fail(GCSPH_EINVAL, "null %s[%d]", name, d + 1);
    out->p[d] = src[d];
  }
  return GCSPH_OK;
}

// the reference's dot product (no contraction) ...
template <int D>
__device__ inline double dotp(const double* a, const double* b) {
  double s = a[0] * b[0];
#pragma unroll
  for (int d = 1; d < D; ++d) s = s + a[d] * b[d];
  return s;
}

// ... and the fused one of the summed terms
template <int D>
__device__ inline double dotf(const double* a, const double* b) {
  double s = a[0] * b[0];
#pragma unroll
  for (int d = 1; d < D; ++d) s = fma(a[d], b[d], s);
  return s;
}

// whether x's exponent lies in a range where the corrected approximations
// hold (2^-900 .. 2^900); zeros, denormals, infinities and NaN take the IEEE
// operations
__device__ inline bool mid_range(double x) {
  return ((unsigned)(dbits(x) >> 32) & 0x7fffffffu) - 0x07b00000u < 0x70800000u;
}
__device__ inline double rcp_pair(double x) { return mid_range(x) ? rcp_nr(x) : 1.0 / x; }
__device__ inline double sqrt_pair(double x) { return mid_range(x) ? sqrt_nr(x) : sqrt(x); }

__device__ inline bool pair_at(const int32_t* pairs, int64_t p, int64_t* i, int64_t* j) {
  int32_t a = pairs[2 * p], b = pairs[2 * p + 1];
  *i = (int64_t)a - 1;
  *j = (int64_t)b - 1;
  return a != 0;
}

// A summed term over the pair list.  F: take(pt of i, pt of j) says whether a
// pair has the term, run(p, i, j) adds it.  QUEUE: a warp's FP64 instruction
// costs the same for one active lane as for 32, and in a tank most lanes hold
// pairs without the term (walls); each warp collects the pairs of its chunks
// that have it and runs 32 at a time.  A list of about one chunk a warp has
// nothing to collect and is run as it comes, and so are the terms that gained
// nothing.  (10.5M pairs of a 3-D tank, 179k particles of them 50k fluid,
// without and with the queue: ∂v∂tpF! 504 and 388 us, sph∑W! 384 and 310,
// ∂v∂t_visc! 345 and 281, fbmolforce! 374 and 223, ∂v∂t_av! 265 and 263, ∂v∂t! 198
// and 180; ∂ρ∂tDDT! 478 and 485, xsphcorr! 151 and 164.)
constexpr int PW = PTPB / 32;
template <class F, bool QUEUE>
__global__ void __launch_bounds__(PTPB) k_pair_term(int64_t P, const int32_t* __restrict__ pairs, const F f) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if constexpr (!QUEUE) {
    const int64_t p = (int64_t)blockIdx.x * PTPB + threadIdx.x;
    if (p >= P) return;
    const int32_t a = pairs[2 * p], b = pairs[2 * p + 1];
    if (a > 0 && f.take(f.pt[a - 1], f.pt[b - 1])) f.run(p, (int64_t)a - 1, (int64_t)b - 1);
    return;
  }
  __shared__ int64_t s_q[PW][64];  // at most 31 waiting and 32 new ones
  int64_t* q = s_q[w];
  int cnt = 0;
  const int64_t nchunk = (P + 31) / 32, step = (int64_t)gridDim.x * PW;
  int64_t ch = (int64_t)blockIdx.x * PW + w;
  bool more;
  do {
    more = ch < nchunk;
    const int64_t p = ch * 32 + lane;
    bool on = false;
    if (p < P) {
      const int32_t a = pairs[2 * p], b = pairs[2 * p + 1];
      on = a > 0 && f.take(f.pt[a - 1], f.pt[b - 1]);
    }
    const unsigned bal = __ballot_sync(0xffffffffu, on);
    if (on) q[cnt + __popc(bal & ((1u << lane) - 1u))] = p;
    cnt += __popc(bal);
    __syncwarp();
    // a full warp's worth, or after the last chunk what is left (under 32)
    const int base = cnt >= 32 ? cnt - 32 : (more ? cnt : 0);
    if (base + lane < cnt) {
      const int64_t u = q[base + lane];
      f.run(u, (int64_t)pairs[2 * u] - 1, (int64_t)pairs[2 * u + 1] - 1);
    }
    cnt = base;
    __syncwarp();
    ch += step;
  } while (more);
}

template <class F>
static int launch_pair_term(int64_t P, const int32_t* pairs, const F& f, cudaStream_t st) {
  if constexpr (F::QUEUE) {
    // the queue form's blocks stay resident: as many as fit
    static int64_t grid = 0;
    if (grid == 0) {
      int dev = 0, sms = 0, per = 0;
      GC_CUDA(cudaGetDevice(&dev));
      GC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
      GC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pair_term<F, true>, PTPB, 0));
      grid = (int64_t)sms * (per > 0 ? per : 1);
    }
    if (P > 2 * grid * PTPB) {
      k_pair_term<F, true><<<(unsigned)grid, PTPB, 0, st>>>(P, pairs, f);
      GC_LAUNCHED();
      return GCSPH_OK;
    }
  }
  k_pair_term<F, false><<<nblocks(P, PTPB), PTPB, 0, st>>>(P, pairs, f);
  GC_LAUNCHED();
  return GCSPH_OK;
}

template <int D>
__device__ inline void pair_dx(const V3& x, int64_t i, int64_t j, double* dx) {
#pragma unroll
  for (int d = 0; d < D; ++d) dx[d] = x.p[d][i] - x.p[d][j];
}
template <int D>
__device__ inline void scatter_pm(const W3& a, int64_t i, int64_t j, const double* f) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    atomicAdd(&a.p[d][i], f[d]);
    atomicAdd(&a.p[d][j], -f[d]);
  }
}

// kernel_sphW! (:84-100) and kernel_sph∇W! (:196-213)
template <int D, int GRAD>
__global__ void k_fn_w(int64_t P, const int32_t* __restrict__ pairs, V3 x, double Hinv, double nn,
                       double* __restrict__ W, W3 gW) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  int64_t i, j;
  if (!pair_at(pairs, p, &i, &j)) return;
  double dx[D];
#pragma unroll
  for (int d = 0; d < D; ++d) dx[d] = x.p[d][i] - x.p[d][j];
  double r = sqrt(dotp<D>(dx, dx));
  double u = r * Hinv;
  if (GRAD) {
    double dwk_r = wc2_dw(u, nn) / r;
#pragma unroll
    for (int d = 0; d < D; ++d) gW.p[d][p] = dx[d] * dwk_r;
  } else {
    W[p] = wc2_w(u, nn);
  }
}

// kernel_sph∑W! (:139-156), kernel_sph∑∇W! (:332-359).  nn: the norm of 𝒲, or
// of d𝒲 times -20 H⁻¹ (d𝒲/r = nn (1 - u)^3, u / r = H⁻¹)
template <int D, int GRAD>
struct TermSumW {
  static constexpr bool QUEUE = true;
  V3 x;
  double Hinv, nn;
  const int32_t* pt;
  double* sumW;
  W3 sg;
  __device__ bool take(int pi, int pj) const { return (pi > 0) == (pj > 0); }
  __device__ void run(int64_t, int64_t i, int64_t j) const {
    double dx[D];
    pair_dx<D>(x, i, j, dx);
    const double r2 = dotf<D>(dx, dx);
    const double u = sqrt_pair(r2) * Hinv;
    // (a NaN distance adds 0 to ∑W and NaN to ∑∇W, an infinite one NaN to ∑∇W)
    if (GRAD ? u >= 1.0 && r2 < INFINITY : !(u < 1.0)) return;
    const double t = u < 1.0 ? 1.0 - u : 0.0, t2 = t * t;
    if (GRAD) {
      const double dwk_r = r2 > 0.0 ? nn * (t2 * t) : NAN;  // the reference's d𝒲(0)/0
      double g[D];
#pragma unroll
      for (int d = 0; d < D; ++d) g[d] = dx[d] * dwk_r;
      scatter_pm<D>(sg, i, j, g);
    } else {
      const double w = fma(4.0, u, 1.0) * (t2 * t2) * nn;
      atomicAdd(&sumW[i], w);
      atomicAdd(&sumW[j], w);
    }
  }
};

// kernel_∂ρ∂tDDT! (:571-631)
template <int D>
struct TermDDT {
  static constexpr bool QUEUE = false;
  V3 gW, v, x;
  const double* rho;
  double eta2, m0, rho0, ginv, DDTkhm0, DDTgz;
  int gamma;
  const int32_t* pt;
  double* out;
  __device__ bool take(int pi, int pj) const { return pi > 0 && pj > 0; }
  __device__ void run(int64_t p, int64_t i, int64_t j) const {
    double dx[D], dv[D], gw[D];
    pair_dx<D>(x, i, j, dx);
    pair_dx<D>(v, i, j, dv);
#pragma unroll
    for (int d = 0; d < D; ++d) gw[d] = gW.p[d][p];
    const double ri = rho[i], rj = rho[j];
    const int pi = pt[i], pj = pt[j];
    double si = m0 * dotf<D>(dv, gw), sj = si;
    if (pi > 1 || pj > 1) {
      const double com = DDTkhm0 * -dotf<D>(dx, gw) * rcp_pair(dotf<D>(dx, dx) + eta2);
      const double ez = DDTgz * dx[1], drr = rj - ri;
      if (pi > 1) {
        const double d = fma(-rho0, pf7m1_fast(ez, ginv, gamma), drr);
        si = fma(d * com, rcp_pair(rj), si);
      }
      if (pj > 1) {
        const double d = fma(-rho0, pf7m1_fast(-ez, ginv, gamma), -drr);
        sj = fma(d * com, rcp_pair(ri), sj);
      }
    }
    atomicAdd(&out[i], si);
    atomicAdd(&out[j], sj);
  }
};

__global__ void k_fn_pressure(int64_t N, const double* __restrict__ rho, int gamma, double rho0, double P0,
                              const int32_t* __restrict__ pt, double* __restrict__ P) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) P[i] = eos(rho[i], gamma, rho0, P0, pt[i]);
}

// kernel_∂v∂t! (:750-776)
template <int D>
struct TermPress {
  static constexpr bool QUEUE = true;
  V3 gW;
  const double* Pr;
  const double* rho;
  double m0;
  const int32_t* pt;
  W3 a;
  __device__ bool take(int pi, int pj) const { return pi * pj > 0; }
  __device__ void run(int64_t p, int64_t i, int64_t j) const {
    const double s = -m0 * (Pr[i] + Pr[j]) * rcp_pair(rho[i] * rho[j]);
    double f[D];
#pragma unroll
    for (int d = 0; d < D; ++d) f[d] = s * gW.p[d][p];
    scatter_pm<D>(a, i, j, f);
  }
};

// kernel_∂v∂t_av! (:863-901): -Π m₀ = avk (Δv·Δx) / ((r² + η²)(ρi + ρj)), avk = 2 α c₀ h m₀
template <int D>
struct TermAv {
  static constexpr bool QUEUE = true;
  V3 gW, x, v;
  const double* rho;
  double eta2, avk;
  const int32_t* pt;
  W3 a;
  __device__ bool take(int pi, int pj) const { return pi > 0 && pj > 0; }
  __device__ void run(int64_t p, int64_t i, int64_t j) const {
    double dx[D], dv[D];
    pair_dx<D>(x, i, j, dx);
    pair_dx<D>(v, i, j, dv);
    const double cond = dotf<D>(dv, dx);
    if (!(cond < 0.0)) return;
    const double s = avk * cond * rcp_pair((dotf<D>(dx, dx) + eta2) * (rho[i] + rho[j]));
    double f[D];
#pragma unroll
    for (int d = 0; d < D; ++d) f[d] = s * gW.p[d][p];
    scatter_pm<D>(a, i, j, f);
  }
};

// kernel_∂v∂t_visc! (:962-991), nu4 = 4 ν m₀
template <int D>
struct TermVisc {
  static constexpr bool QUEUE = true;
  V3 gW, v, x;
  const double* rho;
  double eta2, nu4;
  const int32_t* pt;
  W3 a;
  __device__ bool take(int pi, int pj) const { return pi > 0 && pj > 0; }
  __device__ void run(int64_t p, int64_t i, int64_t j) const {
    double dx[D], dv[D], gw[D], f[D];
    pair_dx<D>(x, i, j, dx);
    pair_dx<D>(v, i, j, dv);
#pragma unroll
    for (int d = 0; d < D; ++d) gw[d] = gW.p[d][p];
    const double nt = nu4 * dotf<D>(dx, gw) * rcp_pair((rho[i] + rho[j]) * (dotf<D>(dx, dx) + eta2));
#pragma unroll
    for (int d = 0; d < D; ++d) f[d] = nt * dv[d];
    scatter_pm<D>(a, i, j, f);
  }
};

template <int D>
__global__ void k_fn_grav(int64_t N, double g, W3 a) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
#pragma unroll
  for (int d = 0; d < D; ++d) a.p[d][i] = a.p[d][i] - (d == 1 ? g : 0.0);
}

// kernel_fbmolforce! (:1885-1913).  Lattice walls hold pairs at exactly r₀: the
// distance and its compare are the reference's to the bit (past r2cut =
// r₀² (1 + 1e-6) it fails for certain)
template <int D>
struct TermWall {
  static constexpr bool QUEUE = true;
  V3 x;
  double dd, r0, eta2, r2cut;
  const int32_t* pt;
  W3 a;
  __device__ bool take(int pi, int pj) const { return (pi > 0) != (pj > 0); }
  __device__ void run(int64_t, int64_t i, int64_t j) const {
    double dx[D];
    pair_dx<D>(x, i, j, dx);
    const double r2 = dotp<D>(dx, dx);
    if (r2 > r2cut) return;
    const double r = sqrt(r2);
    if (!(r < r0)) return;
    const double q = r0 * rcp_pair(r + eta2);
    const double q2 = q * q, q4 = q2 * q2, q8 = q4 * q4, q12 = q8 * q4;
    const double Fc = dd * (q12 - q4) * rcp_pair(r2 + eta2);
    double f[D];
#pragma unroll
    for (int d = 0; d < D; ++d) f[d] = dx[d] * Fc;
    scatter_pm<D>(a, i, j, f);
  }
};

// kernel_∂v∂tpF! (:1382-1409): pfk2 = 2/(2h)², hp1 = 0.1h, C: pf_cos_coef of s/m₀
template <int D>
struct TermTension {
  static constexpr bool QUEUE = true;
  V3 x;
  double twoh, pfk2, hp1;
  const int32_t* pt;
  W3 a;
  double C[PF_COS_N];
  __device__ bool take(int pi, int pj) const { return pi > 0 && pj > 0; }
  __device__ void run(int64_t, int64_t i, int64_t j) const {
    double dx[D];
    pair_dx<D>(x, i, j, dx);
    const double r2 = dotf<D>(dx, dx);
    const double r = sqrt_pair(r2);
    if (!(r < twoh)) return;
    const double scos = pf_cos(r2, pfk2, C) * rcp_pair(r + hp1);
    double f[D];
#pragma unroll
    for (int d = 0; d < D; ++d) f[d] = scos * dx[d];
    scatter_pm<D>(a, i, j, f);
  }
};

__global__ void k_fn_update_rho(int64_t N, double* __restrict__ rho, const double* __restrict__ drho, double dt,
                                double rho0, const int32_t* __restrict__ pt) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double r = rho[i] + drho[i] * dt;
  if (r < rho0 && pt[i] < 0) r = rho0;
  rho[i] = r;
}

template <int D>
__global__ void k_fn_update_v(int64_t N, W3 v, V3 a, double dt, const int32_t* __restrict__ pt) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N || !(pt[i] > 1)) return;
#pragma unroll
  for (int d = 0; d < D; ++d) v.p[d][i] = v.p[d][i] + a.p[d][i] * dt;
}

template <int D>
__global__ void k_fn_update_x(int64_t N, W3 x, V3 v, double dt) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
#pragma unroll
  for (int d = 0; d < D; ++d) x.p[d][i] = x.p[d][i] + v.p[d][i] * dt;
}

// kernel_symplectic_update! (:1204-1245)
template <int D>
__global__ void k_fn_symplectic(int64_t N, double* __restrict__ rho, double* __restrict__ rhoh, W3 v, W3 vh, W3 x,
                                W3 xh, const double* __restrict__ drho, V3 a, double dt, W3 cdx, double rho0,
                                const int32_t* __restrict__ pt) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double epsi = -(drho[i] / rhoh[i]) * dt;
  double rv = rho[i] * (2.0 - epsi) / (2.0 + epsi);
  if (rv < rho0 && pt[i] <= 1) rv = rho0;
  rhoh[i] = rv;
  rho[i] = rv;
  double ml = pt[i] > 1 ? 1.0 : 0.0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    double vv = v.p[d][i];
    double nv = vv + a.p[d][i] * dt * ml;
    vh.p[d][i] = nv;
    v.p[d][i] = nv;
    double ddx = (vv + nv) * 0.5 * dt;
    cdx.p[d][i] = cdx.p[d][i] + ddx;
    double xv = x.p[d][i] + ddx;
    xh.p[d][i] = xv;
    x.p[d][i] = xv;
  }
}

__device__ inline double jmin(double a, double b) { return (a != a || b != b) ? (a + b) : fmin(a, b); }
__device__ inline double jmax(double a, double b) { return (a != a || b != b) ? (a + b) : fmax(a, b); }

// kernel_dpcreg! (:1500-1553)
template <int D>
__global__ void k_fn_dpc(int64_t P, W3 buf, V3 v, const double* __restrict__ rho, const double* __restrict__ Pr,
                         const int32_t* __restrict__ pairs, V3 x, double l0inv, double nW, double whinv, double Pmin,
                         double Pmax, double dt, double lambda, double kernlim, double eta2,
                         const int32_t* __restrict__ pt) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  int64_t i, j;
  if (!pair_at(pairs, p, &i, &j)) return;
  if (!(pt[i] > 0 && pt[j] > 0)) return;
  double dx[D], dv[D], f[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    dx[d] = x.p[d][i] - x.p[d][j];
    dv[d] = v.p[d][i] - v.p[d][j];
  }
  double ri = rho[i], rj = rho[j];
  double r2 = dotp<D>(dx, dx);
  double r = sqrt(r2);
  double u = r * l0inv;
  double w = wc2_w(u, nW);
  double chi = sqrt(w * whinv);
  double k = u < kernlim ? 1.0 : chi;
  double Pb = chi * jmax(jmin(lambda * fabs(Pr[i] + Pr[j]), lambda * Pmax), Pmin);
  double vr = dotp<D>(dv, dx);
  if (vr < 0.0) {
    double vrdr = vr / (r2 + eta2);
#pragma unroll
    for (int d = 0; d < D; ++d) f[d] = k * (-vrdr * dx[d]);
  } else {
    double tvar = 2.0 * dt * Pb / ((ri + rj) * (r2 + eta2));
#pragma unroll
    for (int d = 0; d < D; ++d) f[d] = tvar * dx[d];
  }
  scatter_pm<D>(buf, i, j, f);
}

template <int D>
__global__ void k_fn_update_dpc(int64_t N, W3 v, W3 x, V3 buf, double dt, const int32_t* __restrict__ pt) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N || !(pt[i] > 1)) return;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    v.p[d][i] = v.p[d][i] + buf.p[d][i];
    x.p[d][i] = x.p[d][i] + buf.p[d][i] * dt;
  }
}

// kernel_xsphcorr! (:1757-1779), xc = 2 m₀ ε
template <int D>
struct TermXsph {
  static constexpr bool QUEUE = false;
  V3 v;
  const double* W;
  const double* rho;
  double xc;
  const int32_t* pt;
  W3 buf;
  __device__ bool take(int pi, int pj) const { return pi > 1 && pj > 1; }
  __device__ void run(int64_t p, int64_t i, int64_t j) const {
    const double xs = xc * W[p] * rcp_pair(rho[i] + rho[j]);
    double f[D];
#pragma unroll
    for (int d = 0; d < D; ++d) f[d] = (v.p[d][j] - v.p[d][i]) * xs;
    scatter_pm<D>(buf, i, j, f);
  }
};

template <int D>
__global__ void k_fn_update_xsph(int64_t N, W3 x, V3 buf, double dt, const int32_t* __restrict__ pt) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N || !(pt[i] > 1)) return;
#pragma unroll
  for (int d = 0; d < D; ++d) x.p[d][i] = x.p[d][i] + buf.p[d][i] * dt;
}

// kernel_cspmcorr_1! / _2! (:1693-1719)
__global__ void k_fn_cspm1(int64_t P, double* __restrict__ s1, double* __restrict__ s2, const double* __restrict__ W,
                           const double* __restrict__ rho, double m0, const int32_t* __restrict__ pairs,
                           const int32_t* __restrict__ pt) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  int64_t i, j;
  if (!pair_at(pairs, p, &i, &j)) return;
  if (!(pt[i] > 0 && pt[j] > 0)) return;
  double w = W[p];
  atomicAdd(&s1[i], m0 * w);
  atomicAdd(&s2[i], w * m0 / rho[j]);
  atomicAdd(&s1[j], m0 * w);
  atomicAdd(&s2[j], w * m0 / rho[i]);
}
__global__ void k_fn_cspm2(int64_t N, double* __restrict__ rho, const double* __restrict__ s1,
                           const double* __restrict__ s2) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double nr = s1[i] / s2[i];
  if (!isnan(nr)) rho[i] = nr;
}

// kernel_Δt_stepping_norm! / kernel_Δt_stepping! + the two maxima
template <int D>
__global__ void k_fn_dt(int64_t N, V3 a, V3 v, V3 x, double h, double eta2, unsigned long long* out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double am = 0.0, vm = 0.0;
  if (i < N) {
    double av[D], vv[D], pp[D];
#pragma unroll
    for (int d = 0; d < D; ++d) { av[d] = a.p[d][i]; vv[d] = v.p[d][i]; pp[d] = x.p[d][i]; }
    am = sqrt(dotp<D>(av, av));
    vm = fabs(h * dotp<D>(vv, pp) / (dotp<D>(pp, pp) + eta2));
  }
  am = warp_max(am);
  vm = warp_max(vm);
  if ((threadIdx.x & 31) == 0) {
    atomic_max_pos(&out[0], am);
    atomic_max_pos(&out[1], vm);
  }
}

}  // namespace gcsph

using namespace gcsph;

#define CHECK_D(D) \
  if ((D) != 2 && (D) != 3) return fail(GCSPH_EINVAL, "wrong dimention: D=%d (2 or 3)", (int)(D))
#define CHECK_PAIRS(P, pairs) \
  if ((P) < 0 || ((P) > 0 && !(pairs))) return fail(GCSPH_EINVAL, "bad pair list")
#define FINISH(st)                                \
  do {                                            \
    GC_LAUNCHED();                                \
    GC_CUDA(cudaStreamSynchronize((st)));         \
    return GCSPH_OK;                              \
  } while (0)
// a summed term over the pairs, then the wait that ends the call
#define TERM(D, ST, F2, F3)                                                                        \
  do {                                                                                             \
    const int _rc = (D) == 2 ? launch_pair_term(P, pairs, F2, (ST)) : launch_pair_term(P, pairs, F3, (ST)); \
    if (_rc) return _rc;                                                                           \
    GC_CUDA(cudaStreamSynchronize((ST)));                                                          \
    return GCSPH_OK;                                                                               \
  } while (0)
#define DISPATCH(D, KER, GRID, ST, ...)                                  \
  do {                                                                   \
    if ((D) == 2) KER<2><<<(GRID), PTPB, 0, (ST)>>>(__VA_ARGS__);        \
    else KER<3><<<(GRID), PTPB, 0, (ST)>>>(__VA_ARGS__);                 \
  } while (0)

extern "C" {

double gcsph_dpckernlim(int32_t D) {
  // find_zero(x -> 1 - W(k, x, 1), 0.5): bisection on [0, 1] to adjacent doubles
  double nW = D == 2 ? wc2_norm_w<2>(1.0) : wc2_norm_w<3>(1.0);
  double lo = 0.0, hi = 1.0;
  double flo = 1.0 - wc2_w(lo, nW);
  for (int it = 0; it < 2000; ++it) {
    double mid = lo + (hi - lo) * 0.5;
    if (mid <= lo || mid >= hi) break;
    double fm = 1.0 - wc2_w(mid, nW);
    if (fm == 0.0) return mid;
    if ((fm < 0.0) == (flo < 0.0)) {
      lo = mid;
      flo = fm;
    } else {
      hi = mid;
    }
  }
  double fl = fabs(1.0 - wc2_w(lo, nW)), fh = fabs(1.0 - wc2_w(hi, nW));
  return fl <= fh ? lo : hi;
}

int gcsph_sphW(int32_t D, int64_t N, int64_t P, const int32_t* pairs, const double* const* x_dev, double Hinv,
               double* W, void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  V3 x;
  int rc = vec_in(D, x_dev, &x, "x");
  if (rc) return rc;
  if (!W) return fail(GCSPH_EINVAL, "null W");
  if (P == 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  double nn = D == 2 ? wc2_norm_w<2>(Hinv) : wc2_norm_w<3>(Hinv);
  W3 none{};
  if (D == 2) k_fn_w<2, 0><<<nblocks(P, PTPB), PTPB, 0, st>>>(P, pairs, x, Hinv, nn, W, none);
  else k_fn_w<3, 0><<<nblocks(P, PTPB), PTPB, 0, st>>>(P, pairs, x, Hinv, nn, W, none);
  (void)N;
  FINISH(st);
}

int gcsph_sphgradW(int32_t D, int64_t N, int64_t P, const int32_t* pairs, const double* const* x_dev, double Hinv,
                   double* const* gW_dev, void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  V3 x;
  W3 g;
  int rc = vec_in(D, x_dev, &x, "x");
  if (!rc) rc = vec_out(D, gW_dev, &g, "gradW");
  if (rc) return rc;
  if (P == 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  double nn = D == 2 ? wc2_norm_dw<2>(Hinv) : wc2_norm_dw<3>(Hinv);
  if (D == 2) k_fn_w<2, 1><<<nblocks(P, PTPB), PTPB, 0, st>>>(P, pairs, x, Hinv, nn, nullptr, g);
  else k_fn_w<3, 1><<<nblocks(P, PTPB), PTPB, 0, st>>>(P, pairs, x, Hinv, nn, nullptr, g);
  (void)N;
  FINISH(st);
}

int gcsph_sphsumW(int32_t D, int64_t N, int64_t P, const int32_t* pairs, const double* const* x_dev, double Hinv,
                  const int32_t* pt, double* sumW, void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  V3 x;
  int rc = vec_in(D, x_dev, &x, "x");
  if (rc) return rc;
  if (!pt || !sumW) return fail(GCSPH_EINVAL, "null argument");
  if (P == 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  double nn = D == 2 ? wc2_norm_w<2>(Hinv) : wc2_norm_w<3>(Hinv);
  W3 none{};
  (void)N;
  TERM(D, st, (TermSumW<2, 0>{x, Hinv, nn, pt, sumW, none}), (TermSumW<3, 0>{x, Hinv, nn, pt, sumW, none}));
}

int gcsph_sphsumgradW(int32_t D, int64_t N, int64_t P, const int32_t* pairs, const double* const* x_dev, double Hinv,
                      const int32_t* pt, double* const* sumgW_dev, void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  V3 x;
  W3 g;
  int rc = vec_in(D, x_dev, &x, "x");
  if (!rc) rc = vec_out(D, sumgW_dev, &g, "sumgradW");
  if (rc) return rc;
  if (!pt) return fail(GCSPH_EINVAL, "null ptype");
  if (P == 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  double nn = -20.0 * (D == 2 ? wc2_norm_dw<2>(Hinv) : wc2_norm_dw<3>(Hinv)) * Hinv;
  (void)N;
  TERM(D, st, (TermSumW<2, 1>{x, Hinv, nn, pt, nullptr, g}), (TermSumW<3, 1>{x, Hinv, nn, pt, nullptr, g}));
}

int gcsph_drhodt_ddt(int32_t D, int64_t N, int64_t P, const int32_t* pairs, const double* const* gW_dev,
                     const double* rho, const double* const* v_dev, const double* const* x_dev, double h, double m0,
                     double rho0, double c0, int32_t gamma, double g, double delta, const int32_t* pt, double* out,
                     void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  V3 gw, v, x;
  int rc = vec_in(D, gW_dev, &gw, "gradW");
  if (!rc) rc = vec_in(D, v_dev, &v, "v");
  if (!rc) rc = vec_in(D, x_dev, &x, "x");
  if (rc) return rc;
  if (!rho || !pt || !out) return fail(GCSPH_EINVAL, "null argument");
  if (gamma <= 0) return fail(GCSPH_EINVAL, "gamma must be a positive integer");
  cudaStream_t st = (cudaStream_t)stream;
  GC_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * (size_t)N, st));
  double eta2 = (0.1 * h) * (0.1 * h);
  double ginv = 1.0 / (double)gamma;
  double DDTkh = 2.0 * h * delta * c0;
  double Cb = (c0 * c0 * rho0) * ginv;
  double DDTgz = rho0 * g / Cb;
  if (P > 0)
    TERM(D, st, (TermDDT<2>{gw, v, x, rho, eta2, m0, rho0, ginv, DDTkh * m0, DDTgz, gamma, pt, out}),
         (TermDDT<3>{gw, v, x, rho, eta2, m0, rho0, ginv, DDTkh * m0, DDTgz, gamma, pt, out}));
  GC_CUDA(cudaStreamSynchronize(st));
  return GCSPH_OK;
}

int gcsph_pressure(int64_t N, const double* rho, double c0, int32_t gamma, double rho0, const int32_t* pt, double* P,
                   void* stream) {
  if (!rho || !pt || !P) return fail(GCSPH_EINVAL, "null argument");
  if (gamma <= 0) return fail(GCSPH_EINVAL, "gamma must be a positive integer");
  if (N <= 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  double P0 = c0 * c0 * rho0 / (double)gamma;
  k_fn_pressure<<<nblocks(N, PTPB), PTPB, 0, st>>>(N, rho, gamma, rho0, P0, pt, P);
  FINISH(st);
}

int gcsph_dvdt(int32_t D, int64_t N, int64_t P, const int32_t* pairs, const double* const* gW_dev, const double* Pr,
               double m0, const double* rho, const int32_t* pt, double* const* a_dev, void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  V3 gw;
  W3 a;
  int rc = vec_in(D, gW_dev, &gw, "gradW");
  if (!rc) rc = vec_out(D, a_dev, &a, "a");
  if (rc) return rc;
  if (!Pr || !rho || !pt) return fail(GCSPH_EINVAL, "null argument");
  if (P == 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  (void)N;
  TERM(D, st, (TermPress<2>{gw, Pr, rho, m0, pt, a}), (TermPress<3>{gw, Pr, rho, m0, pt, a}));
}

int gcsph_dvdt_av(int32_t D, int64_t N, int64_t P, const int32_t* pairs, const double* const* gW_dev,
                  const double* const* x_dev, double h, const double* rho, double alpha, const double* const* v_dev,
                  double c0, double m0, const int32_t* pt, double* const* a_dev, void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  V3 gw, x, v;
  W3 a;
  int rc = vec_in(D, gW_dev, &gw, "gradW");
  if (!rc) rc = vec_in(D, x_dev, &x, "x");
  if (!rc) rc = vec_in(D, v_dev, &v, "v");
  if (!rc) rc = vec_out(D, a_dev, &a, "a");
  if (rc) return rc;
  if (!rho || !pt) return fail(GCSPH_EINVAL, "null argument");
  if (P == 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  double eta2 = (0.1 * h) * (0.1 * h);
  const double avk = 2.0 * alpha * c0 * h * m0;
  (void)N;
  TERM(D, st, (TermAv<2>{gw, x, v, rho, eta2, avk, pt, a}), (TermAv<3>{gw, x, v, rho, eta2, avk, pt, a}));
}

int gcsph_dvdt_visc(int32_t D, int64_t N, int64_t P, const int32_t* pairs, const double* const* gW_dev,
                    const double* const* v_dev, const double* rho, const double* const* x_dev, double h, double m0,
                    double nu, const int32_t* pt, double* const* a_dev, void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  V3 gw, x, v;
  W3 a;
  int rc = vec_in(D, gW_dev, &gw, "gradW");
  if (!rc) rc = vec_in(D, x_dev, &x, "x");
  if (!rc) rc = vec_in(D, v_dev, &v, "v");
  if (!rc) rc = vec_out(D, a_dev, &a, "a");
  if (rc) return rc;
  if (!rho || !pt) return fail(GCSPH_EINVAL, "null argument");
  if (P == 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  double eta2 = (0.1 * h) * (0.1 * h);
  const double nu4 = 4.0 * nu * m0;
  (void)N;
  TERM(D, st, (TermVisc<2>{gw, v, x, rho, eta2, nu4, pt, a}), (TermVisc<3>{gw, v, x, rho, eta2, nu4, pt, a}));
}

int gcsph_addgrav(int32_t D, int64_t N, double g, double* const* a_dev, void* stream) {
  CHECK_D(D);
  W3 a;
  int rc = vec_out(D, a_dev, &a, "a");
  if (rc) return rc;
  if (N <= 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  DISPATCH(D, k_fn_grav, nblocks(N, PTPB), st, N, g, a);
  FINISH(st);
}

int gcsph_fbmolforce(int32_t D, int64_t N, int64_t P, const int32_t* pairs, const double* const* x_dev, double d,
                     double r0, const int32_t* pt, double* const* a_dev, void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  V3 x;
  W3 a;
  int rc = vec_in(D, x_dev, &x, "x");
  if (!rc) rc = vec_out(D, a_dev, &a, "a");
  if (rc) return rc;
  if (!pt) return fail(GCSPH_EINVAL, "null ptype");
  if (P == 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  double eta2 = 0.01 * (r0 * r0);
  const double cut = r0 * r0 * (1.0 + 1e-6);
  (void)N;
  TERM(D, st, (TermWall<2>{x, d, r0, eta2, cut, pt, a}), (TermWall<3>{x, d, r0, eta2, cut, pt, a}));
}

int gcsph_dvdt_pF(int32_t D, int64_t N, int64_t P, const int32_t* pairs, const double* const* x_dev, double s,
                  double h, double m0, const int32_t* pt, double* const* a_dev, void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  V3 x;
  W3 a;
  int rc = vec_in(D, x_dev, &x, "x");
  if (!rc) rc = vec_out(D, a_dev, &a, "a");
  if (rc) return rc;
  if (!pt) return fail(GCSPH_EINVAL, "null ptype");
  if (P == 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const double twoh = 2.0 * h, pfk2 = 2.0 / (twoh * twoh), hp1 = 0.1 * h;
  (void)N;
  TermTension<2> f2{x, twoh, pfk2, hp1, pt, a, {}};
  TermTension<3> f3{x, twoh, pfk2, hp1, pt, a, {}};
  pf_cos_coef(s / m0, f2.C);
  pf_cos_coef(s / m0, f3.C);
  TERM(D, st, f2, f3);
}

int gcsph_update_rho(int64_t N, double* rho, const double* drho, double dt, double rho0, const int32_t* pt,
                     void* stream) {
  if (!rho || !drho || !pt) return fail(GCSPH_EINVAL, "null argument");
  if (N <= 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  k_fn_update_rho<<<nblocks(N, PTPB), PTPB, 0, st>>>(N, rho, drho, dt, rho0, pt);
  FINISH(st);
}

int gcsph_update_v(int32_t D, int64_t N, double* const* v_dev, const double* const* a_dev, double dt,
                   const int32_t* pt, void* stream) {
  CHECK_D(D);
  W3 v;
  V3 a;
  int rc = vec_out(D, v_dev, &v, "v");
  if (!rc) rc = vec_in(D, a_dev, &a, "a");
  if (rc) return rc;
  if (!pt) return fail(GCSPH_EINVAL, "null ptype");
  if (N <= 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  DISPATCH(D, k_fn_update_v, nblocks(N, PTPB), st, N, v, a, dt, pt);
  FINISH(st);
}

int gcsph_update_x(int32_t D, int64_t N, double* const* x_dev, const double* const* v_dev, double dt, void* stream) {
  CHECK_D(D);
  W3 x;
  V3 v;
  int rc = vec_out(D, x_dev, &x, "x");
  if (!rc) rc = vec_in(D, v_dev, &v, "v");
  if (rc) return rc;
  if (N <= 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  DISPATCH(D, k_fn_update_x, nblocks(N, PTPB), st, N, x, v, dt);
  FINISH(st);
}

int gcsph_symplectic(int32_t D, int64_t N, double* rho, double* rhoh, double* const* v_dev, double* const* vh_dev,
                     double* const* x_dev, double* const* xh_dev, const double* drho, const double* const* a_dev,
                     double dt, double* const* cdx_dev, double rho0, const int32_t* pt, void* stream) {
  CHECK_D(D);
  W3 v, vh, x, xh, cdx;
  V3 a;
  int rc = vec_out(D, v_dev, &v, "v");
  if (!rc) rc = vec_out(D, vh_dev, &vh, "vh");
  if (!rc) rc = vec_out(D, x_dev, &x, "x");
  if (!rc) rc = vec_out(D, xh_dev, &xh, "xh");
  if (!rc) rc = vec_out(D, cdx_dev, &cdx, "cdx");
  if (!rc) rc = vec_in(D, a_dev, &a, "a");
  if (rc) return rc;
  if (!rho || !rhoh || !drho || !pt) return fail(GCSPH_EINVAL, "null argument");
  if (N <= 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  DISPATCH(D, k_fn_symplectic, nblocks(N, PTPB), st, N, rho, rhoh, v, vh, x, xh, drho, a, dt, cdx, rho0, pt);
  FINISH(st);
}

int gcsph_dpcreg(int32_t D, int64_t N, int64_t P, double* const* buf_dev, const double* const* v_dev,
                 const double* rho, const double* Pr, const int32_t* pairs, const double* const* x_dev, double l0,
                 double Pmin, double Pmax, double dt, double lambda, double kernlim, const int32_t* pt,
                 void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  W3 buf;
  V3 v, x;
  int rc = vec_out(D, buf_dev, &buf, "buf");
  if (!rc) rc = vec_in(D, v_dev, &v, "v");
  if (!rc) rc = vec_in(D, x_dev, &x, "x");
  if (rc) return rc;
  if (!rho || !Pr || !pt) return fail(GCSPH_EINVAL, "null argument");
  if (!(l0 > 0)) return fail(GCSPH_EINVAL, "l0 must be > 0");
  cudaStream_t st = (cudaStream_t)stream;
  for (int d = 0; d < D; ++d) GC_CUDA(cudaMemsetAsync(buf.p[d], 0, sizeof(double) * (size_t)N, st));
  double l0inv = 1.0 / l0;
  double nW = D == 2 ? wc2_norm_w<2>(l0inv) : wc2_norm_w<3>(l0inv);
  double whinv = 1.0 / wc2_w(0.5, nW);
  double eta2 = (0.1 * l0) * (0.1 * l0);
  if (P > 0) {
    DISPATCH(D, k_fn_dpc, nblocks(P, PTPB), st, P, buf, v, rho, Pr, pairs, x, l0inv, nW, whinv, Pmin, Pmax, dt,
             lambda, kernlim, eta2, pt);
    GC_LAUNCHED();
  }
  GC_CUDA(cudaStreamSynchronize(st));
  return GCSPH_OK;
}

int gcsph_update_dpcreg(int32_t D, int64_t N, double* const* v_dev, double* const* x_dev,
                        const double* const* buf_dev, double dt, const int32_t* pt, void* stream) {
  CHECK_D(D);
  W3 v, x;
  V3 buf;
  int rc = vec_out(D, v_dev, &v, "v");
  if (!rc) rc = vec_out(D, x_dev, &x, "x");
  if (!rc) rc = vec_in(D, buf_dev, &buf, "buf");
  if (rc) return rc;
  if (!pt) return fail(GCSPH_EINVAL, "null ptype");
  if (N <= 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  DISPATCH(D, k_fn_update_dpc, nblocks(N, PTPB), st, N, v, x, buf, dt, pt);
  FINISH(st);
}

int gcsph_xsphcorr(int32_t D, int64_t N, int64_t P, double* const* buf_dev, const int32_t* pairs, const double* W,
                   const double* rho, const double* const* v_dev, double m0, double eps, const int32_t* pt,
                   void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  W3 buf;
  V3 v;
  int rc = vec_out(D, buf_dev, &buf, "buf");
  if (!rc) rc = vec_in(D, v_dev, &v, "v");
  if (rc) return rc;
  if (!W || !rho || !pt) return fail(GCSPH_EINVAL, "null argument");
  cudaStream_t st = (cudaStream_t)stream;
  for (int d = 0; d < D; ++d) GC_CUDA(cudaMemsetAsync(buf.p[d], 0, sizeof(double) * (size_t)N, st));
  const double xc = 2.0 * m0 * eps;
  if (P > 0) TERM(D, st, (TermXsph<2>{v, W, rho, xc, pt, buf}), (TermXsph<3>{v, W, rho, xc, pt, buf}));
  GC_CUDA(cudaStreamSynchronize(st));
  return GCSPH_OK;
}

int gcsph_update_xsph(int32_t D, int64_t N, double* const* x_dev, const double* const* buf_dev, double dt,
                      const int32_t* pt, void* stream) {
  CHECK_D(D);
  W3 x;
  V3 buf;
  int rc = vec_out(D, x_dev, &x, "x");
  if (!rc) rc = vec_in(D, buf_dev, &buf, "buf");
  if (rc) return rc;
  if (!pt) return fail(GCSPH_EINVAL, "null ptype");
  if (N <= 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  DISPATCH(D, k_fn_update_xsph, nblocks(N, PTPB), st, N, x, buf, dt, pt);
  FINISH(st);
}

int gcsph_cspmcorr(int32_t D, int64_t N, int64_t P, double* const* buf_dev, const double* W, double* rho, double m0,
                   const int32_t* pairs, const int32_t* pt, void* stream) {
  CHECK_D(D);
  CHECK_PAIRS(P, pairs);
  W3 buf;
  int rc = vec_out(D, buf_dev, &buf, "buf");
  if (rc) return rc;
  if (!W || !rho || !pt) return fail(GCSPH_EINVAL, "null argument");
  if (N <= 0) return GCSPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  for (int d = 0; d < D; ++d) GC_CUDA(cudaMemsetAsync(buf.p[d], 0, sizeof(double) * (size_t)N, st));
  if (P > 0) {
    k_fn_cspm1<<<nblocks(P, PTPB), PTPB, 0, st>>>(P, buf.p[0], buf.p[1], W, rho, m0, pairs, pt);
    GC_LAUNCHED();
  }
  k_fn_cspm2<<<nblocks(N, PTPB), PTPB, 0, st>>>(N, rho, buf.p[0], buf.p[1]);
  FINISH(st);
}

int gcsph_dt_stepping(int32_t D, int64_t N, const double* const* a_dev, const double* const* v_dev,
                      const double* const* x_dev, double c0, double h, double CFL, double tmin, double tmax,
                      double* dt_out, void* stream) {
  CHECK_D(D);
  V3 a, v, x;
  int rc = vec_in(D, a_dev, &a, "a");
  if (!rc) rc = vec_in(D, v_dev, &v, "v");
  if (!rc) rc = vec_in(D, x_dev, &x, "x");
  if (rc) return rc;
  if (!dt_out) return fail(GCSPH_EINVAL, "null dt_out");
  if (N <= 0) return fail(GCSPH_EINVAL, "empty problem");
  cudaStream_t st = (cudaStream_t)stream;
  DevBuf tmp;
  if ((rc = tmp.ensure(2 * sizeof(unsigned long long), st, true))) return rc;
  double eta2 = (0.01 * h) * (0.01 * h);
  DISPATCH(D, k_fn_dt, nblocks(N, PTPB), st, N, a, v, x, h, eta2, tmp.as<unsigned long long>());
  GC_LAUNCHED();
  unsigned long long hb[2];
  cudaError_t e = cudaMemcpyAsync(hb, tmp.p, sizeof(hb), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  tmp.release();
  if (e != cudaSuccess) return cuda_fail(e, "dt readback", __FILE__, __LINE__);
  double amax, vmax;
  memcpy(&amax, &hb[0], 8);
  memcpy(&vmax, &hb[1], 8);
  double dt1 = sqrt(h / (3.0 * amax));
  double dt2 = h / (c0 + vmax);
  double dt = CFL * fmin(dt1, dt2);
  dt = fmin(fmax(dt, tmin), tmax);
  *dt_out = dt;
  return GCSPH_OK;
}

}  // extern "C"
