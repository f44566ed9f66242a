// sph_once.cu -- the pair-once split-row passes of the FP64 step (lanes > 1,
// the default).  Compiled with FMA contraction: these passes are FP64-pipe
// bound on GB300 and contraction removes a multiply or an add from every
// fused product-sum; their results are held to the FP64 contract against the
// oracle (within 1e-12, or the reference's own re-association and rounding
// noise), not bit-identity, which the serial row order in sph_step.cu keeps.
#include "sph_step.cuh"

namespace gcsph {

// fbmolforce!, :1891-1901, for a pair with exactly one real side, at
// separation dx: adds Δx Fc to f.  Lattice walls hold pairs at exactly r₀, where
// the last bits of r² and of its root decide: the sum is the reference's (left to
// right, no contraction), and r < r₀ is r² <= fb_r2max.
template <int D>
__device__ inline void fb_pair(const StepConst& c, const double* dx, double* f) {
  double r2 = __dmul_rn(dx[0], dx[0]);
#pragma unroll
  for (int d = 1; d < D; ++d) r2 = __dadd_rn(r2, __dmul_rn(dx[d], dx[d]));
  if (dbits(r2) <= dbits(c.fb_r2max)) {
    const double r = dbits(r2) != 0 ? sqrt_nr(r2) : 0.0;
    const double q = c.fb_r0 * rcp_nr(r + c.fb_eta2);
    const double q2 = q * q, q4 = q2 * q2, q8 = q4 * q4, q12 = q8 * q4;
    const double Fc = c.fb_d * (q12 - q4) * rcp_nr(r2 + c.fb_eta2);
#pragma unroll
    for (int d = 0; d < D; ++d) f[d] += dx[d] * Fc;
  }
}

// Pass A: one thread per pair (k, m), k < m in cell order.  Stage 1 at
// (x, ρ, v, P(ρ)) also writes ∇W, and W in the steps that read it; stage 2
// at (xΔt½, ρΔt½, vΔt½, P(ρΔt½)) with the stage-1 ∇W and fbmolforce! at x.
// The reference's terms,
// src/gpukernels_sph.jl, in their algebraically equal pair-once forms:
//  * m₀∇W = Δx m₀d𝒲/r with m₀d𝒲/r = dWr (1 - u)^3 -- no division by r, and
//    every term's m₀ with it; in stage 1 then Δv·∇W = (Δv·Δx) d𝒲/r and
//    Δx·∇W = r² d𝒲/r;
//  * ∂ρ∂tDDT! (:542-631): both sides share DDTkh m₀ (-Δx·∇W)/(r² + η²);
//  * ∂v∂t! (:740-776) and ∂v∂t_av! (:852-901) as one factor of m₀∇W,
//    -(Pk + Pm)/(ρk ρm) + 2 α c₀ h (Δv·Δx)/((r² + η²)(ρk + ρm));
//  * ∂v∂tpF! (:1373-1409) as one factor of Δx, its cosine from r² (pf_cos).
// The FP64 pipe bounds the pass, so a pair runs only the terms its ptypes
// allow (PairClass), and a warp runs 32 pairs of one class: a warp's FP64
// instruction takes the pipe 16 cycles whatever lanes are active.
enum PairClass {
  PC_FLUID = 0,  // both real, one of them fluid: every term
  PC_WALL = 1,   // both real and no fluid (no δ-SPH term), or both negative (pressure alone)
  PC_MIXED = 2,  // one side real: fbmolforce! alone, and that only within r₀
  PC_NONE = 3    // no term (the walls' inner pairs): stage 1 writes zero slots, stage 2 leaves them
};
__device__ __forceinline__ int pair_class(int ptk, int ptm) {
  const bool rk = ptk > 0, rm = ptm > 0;
  if (rk != rm) return PC_MIXED;
  if (rk) return ptk > 1 || ptm > 1 ? PC_FLUID : PC_WALL;
  return ptk * ptm > 0 ? PC_WALL : PC_NONE;
}

// pair u; in stage 1 a mirror the fill left open is found first: the
// partner's row was not staged when the pair list was written, so it is k's
// position in m's (ascending) row of the finished neighbour list
template <int D, int STAGE>
__device__ __forceinline__ int4 pair_load(const SArr<D>& S, const PairBuf& B, int u) {
  int4 q = B.pq[u];
  if (STAGE == 1 && q.w < 0) {
    int64_t lo = S.rs[q.y], hi = S.rs[q.y + 1];
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (S.nbr[mid] < q.x) lo = mid + 1;
      else hi = mid;
    }
    q.w = (int)lo;
    B.pq[u] = q;
  }
  return q;
}

// -x on the integer pipe
__device__ __forceinline__ double flip(double x) { return __longlong_as_double(dbits(x) ^ (1ll << 63)); }

// A pair past the reach of every term (H, and 2h with ∂v∂tpF!), as a list with
// a skin holds them: its slots, W and ∇W are zero.  Stage 2 takes stage 1's ∇W
// and ∂v∂tpF! at xΔt½.  Such a pair then costs 2 D + 2 FP64 instructions instead
// of 70 to 90, which every pair pays, so make_const sets far_r2 only for lists
// that reach 3% past (break-even: 5% of the pairs).  At a NaN or an infinity in
// what the terms read they are NaN at any distance: a pair at such a separation
// is not far, and once a particle's other values are such (Scal::wild, kept by
// the passes that write them) no pair is.  (Read pair by pair, those values
// cost 1.6% of a call with surface tension, 65k particles in 2-D.)
// (read where it is asked for: held over the loop it took a register more)
__device__ __forceinline__ bool tame(const int* wild) {
  int w;
  asm volatile("ld.global.ca.b32 %0, [%1];" : "=r"(w) : "l"(wild));
  return w == 0;
}
template <int D, int STAGE>
__device__ __forceinline__ bool pair_far(const StepConst& c, const SArr<D>& S, int u, const int4 q) {
  if (STAGE == 2) {
    long long any = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) any |= dbits(S.gWe[d][u]);
    if ((any << 1) != 0) return false;
    if (!c.use_pF) return tame(S.wild);
  }
  const double* const* XP = STAGE == 1 ? S.x : S.xh;
  double dx[D];
#pragma unroll
  for (int d = 0; d < D; ++d) dx[d] = XP[d][q.x] - XP[d][q.y];
  const double r2 = dotD<D>(dx, dx);
  return dbits(r2) > dbits(c.far_r2) && dbits(r2) < dbits((double)INFINITY) && tame(S.wild);
}

template <int D, int STAGE>
__device__ __forceinline__ void pairA_one(const StepConst& c, const SArr<D>& S, const PairBuf& B, int u,
                                          const int4 q, const int ptk, const int ptm) {
  const int k = q.x, m = q.y, e = q.z, me = q.w;
  const bool both = ptk > 0 && ptm > 0;
  const bool press = ptk * ptm > 0;
  double dk = 0.0, dm = 0.0, f[3] = {0.0, 0.0, 0.0};
  if ((ptk > 0) != (ptm > 0)) {
    double dx[D];
#pragma unroll
    for (int d = 0; d < D; ++d) dx[d] = S.x[d][k] - S.x[d][m];
    fb_pair<D>(c, dx, f);
  } else {
    const double* const* XP = STAGE == 1 ? S.x : S.xh;
    const double* const* VP = STAGE == 1 ? S.v : S.vh;
    const double* RP = STAGE == 1 ? S.rho : S.rhoh;
    const double* PP = STAGE == 1 ? S.P1 : S.P2;
    const double* IP = STAGE == 1 ? S.ir : S.irh;
    double dx[D], dv[D], gw[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      dx[d] = XP[d][k] - XP[d][m];
      dv[d] = VP[d][k] - VP[d][m];
    }
    const double r2 = dotD<D>(dx, dx);
    const double cond = dotD<D>(dv, dx);
    const bool r2pos = dbits(r2) != 0;  // r2 is +0 or positive
    double r = 0.0, dr = 0.0, dxgw, dvgw;
    if (STAGE == 1) {
      if (r2pos) r = sqrt_nr(r2);
      const double t = fma(-r, c.Hinv, 1.0);  // 1 - u
      double w = 0.0, dwr = 0.0;
      if ((unsigned long long)dbits(t) - 1ull < (unsigned long long)ONE_BITS) {  // 0 < 1 - u <= 1, and not NaN
        const double t2 = t * t;
        if (c.need_w) w = fma(-4.0, t, 5.0) * (t2 * t2);
        dwr = (t2 * t) * c.dWr;
      }
      if (!r2pos) dwr = NAN;  // the reference's d𝒲(0)/0
      if (c.need_w) {
        // (without 𝒲's norm) in both rows' slots: xsphcorr! and cspmcorr! walk
        // every row (and read the pairs of two real sides only)
        S.We[e] = w;
        S.We[me] = w;
      }
      // stage 2 reads ∇W by pair (the call's ∑∇W is recomputed from the
      // positions at its end)
#pragma unroll
      for (int d = 0; d < D; ++d) {
        gw[d] = dx[d] * dwr;
        S.gWe[d][u] = gw[d];
      }
      dr = dwr;
      dxgw = r2 * dwr;
      dvgw = cond * dwr;
    } else {
#pragma unroll
      for (int d = 0; d < D; ++d) gw[d] = S.gWe[d][u];
      dxgw = dotD<D>(dx, gw);
      dvgw = dotD<D>(dv, gw);
    }
    const double rk = RP[k], rm = RP[m], irk = IP[k], irm = IP[m];
    double sg = press ? -((PP[k] + PP[m]) * (irk * irm)) : 0.0;
    double visc = 0.0;
    if (both) {
      const double s = rk + rm;
      const double ii = rcp_nr(s * (r2 + c.eta2));
      const double g = dxgw * ii;
      dk = dvgw;
      dm = dk;
      if (ptk > 1 || ptm > 1) {
        const double com = -(c.DDTkh * g) * s;
        const double ez = c.DDTgz * dx[1];
        const double drr = rm - rk;
        if (ptk > 1) {
          const double dp = c.rho0 * pf7_fast(ez, c.ginv, c.gamma) - c.rho0;
          dk += (drr - dp) * com * irm;
        }
        if (ptm > 1) {
          const double dn = c.rho0 * pf7_fast(-ez, c.ginv, c.gamma) - c.rho0;
          dm += (-drr - dn) * com * irk;
        }
      }
      if (neg_int(cond)) sg += c.avK * (cond * ii);
      if (c.use_visc) visc = c.visc4 * g;
    }
    const bool pF = c.use_pF && both && (STAGE == 1 ? dbits(r) < dbits(c.twoh) : true);
    double scos = 0.0;
    if (pF) {
      if (STAGE == 2 && r2pos) r = sqrt_nr(r2);
      if (STAGE == 1 || dbits(r) < dbits(c.twoh)) scos = pf_cos(r2, c.pfk2, c.pfc_s) * rcp_nr(r + c.hp1);
    }
    if (STAGE == 1 && c.use_pF) {
      // everything along Δx in one factor
      const double a = fma(sg, dr, scos);
#pragma unroll
      for (int d = 0; d < D; ++d) f[d] = a * dx[d];
    } else {
#pragma unroll
      for (int d = 0; d < D; ++d) f[d] = sg * gw[d];
      if (pF)
#pragma unroll
        for (int d = 0; d < D; ++d) f[d] = fma(scos, dx[d], f[d]);
    }
    if (c.use_visc)
#pragma unroll
      for (int d = 0; d < D; ++d) f[d] = fma(visc, dv[d], f[d]);
  }
  put_slot(B.ce + e, dk, f[0], f[1], f[2]);
  put_slot(B.ce + me, dm, flip(f[0]), flip(f[1]), flip(f[2]));
}

// Pass A over all pairs in chunks of 32 consecutive pairs, one chunk per warp
// at a time, with one block per SM: its threads' registers leave no room for
// a second block, and the grid is the SM count.  Block b
// takes chunks b, b + G, b + 2G, ... (G blocks) and its warp w every NW-th
// of those, so every SM gets the same number of chunks (to one) -- a grid of
// many small blocks leaves some SMs one block more than others -- and
// consecutive chunks of the cell-ordered list, runs of costly fluid pairs or
// of cheap boundary pairs, go to different SMs.
//
// QUEUE: a warp sorts the pairs of its chunks into one short queue per class
// and runs a class whenever 32 of its pairs are waiting, the rest at the end
// (measured: 98k particles in a 3-D tank, 5.5M pairs, stage 1 607 -> 434 us).
// Where a warp has one chunk there is nothing to sort into and the queue only
// adds latency (2-D dam break, 102k pairs: 18.7 us without it, 19.1 with it):
// such lists are run as they come.
//
// Threads: 768 of 80 registers in the direct form.  The queue form does better
// with 640 of 96 (2-D full physics with a skin, 65k particles, a call of ten
// steps: 512 threads 6114 us, 576 6084, 640 6057, 704 6113, 768 6191, 896 6335,
// 1024 6506; 3-D full 24.07, 24.22, 24.02, 24.15, 24.21, 25.45, 25.64 ms): the
// FP64 pipe is about 85% busy from 16 warps on, and fewer registers spill.
template <bool QUEUE>
__host__ __device__ constexpr int pa_tpb() {
  return QUEUE ? 640 : 768;
}
template <int D, int STAGE, bool QUEUE>
__global__ void __launch_bounds__(pa_tpb<QUEUE>(), 1) k_pairA(StepConst c, SArr<D> S, PairBuf B) {
  if (*S.ovf) return;
  constexpr int NW = pa_tpb<QUEUE>() / 32, NC = 3;
  const int np = (int)*B.npair;    // the pair list holds fewer than 2^31
  const int G = gridDim.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nchunk = (np + 31) / 32;
  int64_t ch = blockIdx.x + (int64_t)G * w;
  // pair u's class; a pair without terms is done here
  auto classify = [&](int u, int4& q, int& ptk, int& ptm) {
    q = pair_load<D, STAGE>(S, B, u);
    ptk = S.pt[q.x];
    ptm = S.pt[q.y];
    int cl = pair_class(ptk, ptm);
    bool far = false;
    if (QUEUE && c.far_r2 > 0.0 && (cl == PC_FLUID || cl == PC_WALL)) far = pair_far<D, STAGE>(c, S, (int)u, q);
    if (far) {
      cl = PC_NONE;
      if (STAGE == 1) {
#pragma unroll
        for (int d = 0; d < D; ++d) S.gWe[d][u] = 0.0;
        if (c.need_w) {
          S.We[q.z] = 0.0;
          S.We[q.w] = 0.0;
        }
      }
    }
    if ((STAGE == 1 && cl == PC_NONE) || far) {
      put_slot(B.ce + q.z, 0.0, 0.0, 0.0, 0.0);
      put_slot(B.ce + q.w, 0.0, 0.0, 0.0, 0.0);
    }
    return cl;
  };
  int4 q;
  int ptk, ptm;
  if constexpr (!QUEUE) {
    for (; ch < nchunk; ch += (int64_t)G * NW) {
      const int64_t u = ch * 32 + lane;
      if (u < np && classify((int)u, q, ptk, ptm) != PC_NONE) pairA_one<D, STAGE>(c, S, B, (int)u, q, ptk, ptm);
    }
    return;
  }
  __shared__ int s_q[NW][NC][64];  // at most 31 waiting and 32 new ones
  int cnt[NC] = {0, 0, 0};
  bool more;
  do {
    more = ch < nchunk;
    const int64_t u = ch * 32 + lane;
    const int cl = u < np ? classify((int)u, q, ptk, ptm) : -1;
#pragma unroll
    for (int t = 0; t < NC; ++t) {
      const unsigned bal = __ballot_sync(0xffffffffu, cl == t);
      if (cl == t) s_q[w][t][cnt[t] + __popc(bal & ((1u << lane) - 1u))] = (int)u;
      cnt[t] += __popc(bal);
    }
    __syncwarp();
#pragma unroll 1
    for (int t = 0; t < NC; ++t) {
      // a full warp's worth, or after the last chunk what is left (under 32)
      const int n = t == 0 ? cnt[0] : (t == 1 ? cnt[1] : cnt[2]);
      const int base = n >= 32 ? n - 32 : (more ? n : 0);
      if (base + lane < n) {
        const int v = s_q[w][t][base + lane];
        q = B.pq[v];
        pairA_one<D, STAGE>(c, S, B, v, q, S.pt[q.x], S.pt[q.y]);
      }
      if (t == 0) cnt[0] = base;
      else if (t == 1) cnt[1] = base;
      else cnt[2] = base;
    }
    __syncwarp();
    ch += (int64_t)G * NW;
  } while (more);
}

// Pass B: a block of 32 L threads holds 32 particles, L lanes summing each
// row; the sums go through shared memory to warp 0, which runs the
// per-particle update for all 32 at once.  (Run by each group's lane 0, the
// update's divisions and EOS power would issue on the FP64 pipe with 32 / L
// lanes of a warp active: GB300 issues 2 FP64 thread-instructions per cycle
// per SM, so that costs the full warp's time for a few lanes' work.)
struct RowSums {
  double v[4][32];  // ∂ρ/∂t, then ∂v/∂t, of the block's particles
};

// The four sums of a row over its L lanes.  Each of the first two exchanges
// halves the values a lane still carries instead of summing all four on every
// lane: 2 + 1 adds and one per further level, where a butterfly of all four
// takes 4 log2 L -- at 32 lanes the butterfly cost the FP64 pipe more than
// the row's entries did.  Lane q < 4 ends with the value of index
// 2 (q & 1) + (q >> 1); with L = 2, lane 0 with 0 and 1 and lane 1 with 2 and 3.
template <int L>
__device__ __forceinline__ void lanes_total4(const double* s, int lane, int g, unsigned gm, RowSums& R) {
  const bool b0 = lane & 1, b1 = lane & 2;
  double k0 = b0 ? s[2] : s[0], k1 = b0 ? s[3] : s[1];
  k0 += __shfl_xor_sync(gm, b0 ? s[0] : s[2], 1);
  k1 += __shfl_xor_sync(gm, b0 ? s[1] : s[3], 1);
  if constexpr (L == 2) {
    R.v[2 * lane][g] = k0;
    R.v[2 * lane + 1][g] = k1;
  } else {
    double t = b1 ? k1 : k0;
    t += __shfl_xor_sync(gm, b1 ? k0 : k1, 2);
#pragma unroll
    for (int o = 4; o < L; o <<= 1) t += __shfl_xor_sync(gm, t, o);
    if (lane < 4) R.v[2 * (lane & 1) + (lane >> 1)][g] = t;
  }
}

template <int D, int L>
__device__ __forceinline__ void pairB_sums(const SArr<D>& S, const PairBuf& B, int64_t N, RowSums& R) {
  const int g = threadIdx.x / L, lane = threadIdx.x % L;
  const int64_t k = (int64_t)blockIdx.x * 32 + g;
  if (k < N) {  // whole groups take part
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    const int64_t e1 = S.rs[k + 1];
    int64_t e = S.rs[k] + lane;
    // four entries' loads in flight at a time; each lane adds its entries in
    // row order
    for (; e + 3 * L < e1; e += 4 * L) {
      double v[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) get_slot(B.ce + e + j * L, v[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int d = 0; d < 1 + D; ++d) s[d] += v[j][d];
    }
    for (; e < e1; e += L) {
      double v[4];
      get_slot(B.ce + e, v);
#pragma unroll
      for (int d = 0; d < 1 + D; ++d) s[d] += v[d];
    }
    lanes_total4<L>(s, lane, g, group_mask<L>(), R);
  }
  __syncthreads();
}

// pass B, stage 1: row sums + the three half-step predictors
template <int D, int L>
__global__ void __launch_bounds__(32 * L) k_pairB1(StepConst c, const Scal* __restrict__ sc, int64_t N, SArr<D> S,
                                                   PairBuf B) {
  if (*S.ovf) return;
  __shared__ RowSums R;
  // warp 0 updates the block's 32 particles: their state is loaded before the
  // row sums, so that these loads overlap them (the row sums read only the
  // entry slots)
  const int64_t k = (int64_t)blockIdx.x * 32 + threadIdx.x;
  const bool mine = threadIdx.x < 32 && k < N;
  int ptk = 0;
  double hdt = 0.0, rh0 = 0.0, vh0[D], xh0[D];
  if (mine) {
    ptk = S.pt[k];
    hdt = sc->dt * 0.5;
    rh0 = S.rhoh[k];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      vh0[d] = S.vh[d][k];
      xh0[d] = S.xh[d][k];
    }
  }
  pairB_sums<D, L>(S, B, N, R);
  if (!mine) return;
  double a[D];
#pragma unroll
  for (int d = 0; d < D; ++d) a[d] = R.v[1 + d][threadIdx.x];
  const double drho = R.v[0][threadIdx.x];
  a[1] = a[1] - c.g;
  double rv = rh0 + drho * hdt;
  if (rv < c.rho0 && ptk < 0) rv = c.rho0;
  S.rhoh[k] = rv;
  unsigned top = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    double vh = vh0[d];
    if (ptk > 1) vh = vh + a[d] * hdt;
    S.vh[d][k] = vh;
    S.xh[d][k] = xh0[d] + vh * hdt;
    top = max(top, exponent(vh));
  }
  const double Pk = eos(rv, c.gamma, c.rho0, c.P0, ptk), irk = 1.0 / rv;
  S.P2[k] = Pk;
  S.irh[k] = irk;
  note_wild(S.wild, max(max(top, exponent(rv)), max(exponent(Pk), exponent(irk))));
}

// pass B, stage 2: row sums + symplectic_update! + max |cΔx|; with nb.key
// also the next binning's keys, slots and (last block) cell starts
template <int D, int L>
__global__ void __launch_bounds__(32 * L) k_pairB2(StepConst c, Scal* __restrict__ sc, int64_t N, SArr<D> S,
                                                   PairBuf B, NextBin nb, PosCopy pc) {
  if (*S.ovf) return;  // uniform over the grid, before the barriers below
  __shared__ RowSums R;
  const bool w0 = threadIdx.x < 32;
  const int64_t k = (int64_t)blockIdx.x * 32 + threadIdx.x;
  // warp 0's particles' state, loaded before the row sums so that these
  // loads overlap them (the row sums read only the entry slots)
  const bool mine = w0 && k < N;
  int ptk = 0;
  double dt = 0.0, p2 = 0.0, rh = 0.0, r0 = 0.0, v0[D], cd0[D], x0[D];
  if (mine) {
    ptk = S.pt[k];
    dt = sc->dt;
    p2 = S.P2[k];
    rh = S.rhoh[k];
    r0 = S.rho[k];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      v0[d] = S.v[d][k];
      cd0[d] = S.cdx[d][k];
      x0[d] = S.x[d][k];
    }
  }
  pairB_sums<D, L>(S, B, N, R);
  if (!w0 && !nb.key) return;
  double mc = 0.0;
  if (mine) {
    double a[D], xn[D];
#pragma unroll
    for (int d = 0; d < D; ++d) a[d] = R.v[1 + d][threadIdx.x];
    const double drho = R.v[0][threadIdx.x];
    a[1] = a[1] - c.g;
    S.drho[k] = drho;
    S.Plast[k] = p2;
    const double epsi = -(drho / rh) * dt;
    double rv = r0 * (2.0 - epsi) / (2.0 + epsi);
    if (rv < c.rho0 && ptk <= 1) rv = c.rho0;
    S.rho[k] = rv;
    S.rhoho[k] = rv;
    const double Pk = eos(rv, c.gamma, c.rho0, c.P0, ptk), irk = 1.0 / rv;
    S.P1[k] = Pk;
    S.ir[k] = irk;
    unsigned top = max(exponent(rv), max(exponent(Pk), exponent(irk)));
    const double ml = ptk > 1 ? 1.0 : 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      S.a[d][k] = a[d];
      const double vv = v0[d];
      const double nv = vv + a[d] * dt * ml;
      S.vho[d][k] = nv;
      S.v[d][k] = nv;
      top = max(top, exponent(nv));
      const double ddx = (vv + nv) * 0.5 * dt;
      const double cd = cd0[d] + ddx;
      S.cdx[d][k] = cd;
      mc = fmax(mc, fabs(cd));
      const double xv = x0[d] + ddx;
      S.xho[d][k] = xv;
      S.xo[d][k] = xv;
      xn[d] = xv;
      if (pc.f[0]) pc.f[d][k] = (float)(xv - pc.off[d]);
    }
    note_wild(S.wild, top);
    if (nb.key) {
      const int32_t ck = cell_key_v<D>(xn, nb.g);
      nb.key[k] = ck;
      nb.slot[k] = atomicAdd(&nb.count[ck], 1);
    }
  }
  if (w0) {
    mc = warp_max(mc);
    __syncwarp();
    if (threadIdx.x == 0) atomic_max_pos(&sc->maxcdx, mc);
  }
  if (nb.key) {
    // the whole block takes part: the last one ends the step (k_step_end's
    // work) and scans the next binning's cell starts, then zeroes the counts
    if (last_block_of_grid(&sc->bdone)) {
      if (threadIdx.x == 0) {
        sc->maxcdx = atomicAdd(&sc->maxcdx, 0ull);  // every block's maximum, seen from here
        step_end_body(c, sc);
      }
      block_exclusive_scan<int32_t>(nb.count, nb.cellstart, nb.g.ncell);
      __syncthreads();
      for (int64_t cc = threadIdx.x; cc < nb.g.ncell; cc += blockDim.x) nb.count[cc] = 0;
    }
    return;
  }
  if (threadIdx.x == 0 && c.fold_end) {
    // the last block to finish ends the step (k_step_end's work); only warp
    // 0 of each block writes step state, and its lane 0 signals here
    __threadfence();
    if (atomicAdd(&sc->bdone, 1u) == gridDim.x - 1) {
      __threadfence();
      sc->maxcdx = atomicAdd(&sc->maxcdx, 0ull);  // every block's maximum, seen from here
      step_end_body(c, sc);
      sc->bdone = 0u;
    }
  }
}


// ---------------------------------------------------------------------------
// The gathers of a split-row step and the sums of a call: L lanes walk a
// particle's row, GATHER_U entries of each lane in flight at a time (a row's
// loads depend on its entry's index: at one entry a time these passes waited
// on that chain).  Their FP64 instructions are the second bound, so divisions
// and roots take the same forms as pass A's.
// ---------------------------------------------------------------------------
constexpr int GATHER_U = 4;

// the sums s[0 .. n) of a row over its L lanes, on every lane (lanes_total4's
// exchange, then the owners' values back)
template <int L>
__device__ __forceinline__ void lanes_sum4(double* s, int lane, unsigned gm) {
  const bool b0 = lane & 1, b1 = lane & 2;
  double k0 = b0 ? s[2] : s[0], k1 = b0 ? s[3] : s[1];
  k0 += __shfl_xor_sync(gm, b0 ? s[0] : s[2], 1, L);
  k1 += __shfl_xor_sync(gm, b0 ? s[1] : s[3], 1, L);
  if constexpr (L == 2) {
    s[0] = __shfl_sync(gm, k0, 0, L);
    s[1] = __shfl_sync(gm, k1, 0, L);
    s[2] = __shfl_sync(gm, k0, 1, L);
    s[3] = __shfl_sync(gm, k1, 1, L);
  } else {
    double t = b1 ? k1 : k0;
    t += __shfl_xor_sync(gm, b1 ? k0 : k1, 2, L);
#pragma unroll
    for (int o = 4; o < L; o <<= 1) t += __shfl_xor_sync(gm, t, o, L);
    s[0] = __shfl_sync(gm, t, 0, L);
    s[1] = __shfl_sync(gm, t, 2, L);
    s[2] = __shfl_sync(gm, t, 1, L);
    s[3] = __shfl_sync(gm, t, 3, L);
  }
}

// dpcreg! + update_dpcreg!  (src/gpukernels_sph.jl:1500-1553, :1617-1632).
// W = 0 from u = r / l₀ >= 1 on, so χ = 0, the factor (u >= dpckernlim) is χ
// and Pᵇ = 0: such a pair adds an exact zero to either branch's sum.  l₀ lies
// well under the spacing, so nearly every entry is one of those, and it is
// told apart in FP32 on pass B2's copy of the positions: with R the largest
// |x - offset| component of the particle, the copies of a pair with |Δx| <= l
// differ by at most l + 2^-23 (R + l) per component, so past
// (l + 2^-21 (R + l))² (1 + 2^-20) in FP32 it is beyond l = l₀ (1 + 1e-6).  The
// rest take the FP64 test and terms.  (390k particles, 3-D: the FP64 test of
// every entry cost 1.07 ms a step.)
template <int D, int L>
__global__ void __launch_bounds__(STPB) k_dpc_rows(StepConst c, const Scal* __restrict__ sc, int64_t N, SArr<D> S,
                                                   PosCopy pc) {
  if (*S.ovf) return;
  const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t k = gt / L;
  const int lane = (int)(gt % L);
  if (k >= N) return;  // whole groups leave together
  double sum[4] = {0.0, 0.0, 0.0, 0.0};
  const int ptk = S.pt[k];
  const double Pk = S.P1[k];
  double xk[D], vk[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    xk[d] = S.x[d][k];
    vk[d] = S.v[d][k];
  }
  if (ptk > 0) {
    const double rk = S.rho[k], dt = sc->dt;
    float fk[D];
    double R = 0.0;
    bool nan = false;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      fk[d] = pc.f[d][k];
      R = fmax(R, fabs(xk[d] - pc.off[d]));
      nan |= fk[d] != fk[d];
    }
    const double l = 1.000001 / c.dpc_l0inv;
    const double lim = l + 0x1p-21 * (R + l);
    const float thr = nan ? INFINITY : __double2float_ru(lim * lim * (1.0 + 0x1p-20));
    const int64_t e1 = S.rs[k + 1];
    for (int64_t e = S.rs[k] + lane; e < e1; e += GATHER_U * L) {
      int32_t m[GATHER_U];
      float r2f[GATHER_U];
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) m[j] = e + j * L < e1 ? S.nbr[e + j * L] : (int32_t)k;
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) {
        r2f[j] = 0.f;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          const float df = fk[d] - pc.f[d][m[j]];
          r2f[j] = fmaf(df, df, r2f[j]);
        }
      }
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) {
        if (r2f[j] > thr || m[j] == k) continue;
        const int32_t i = m[j];
        if (!(S.pt[i] > 0)) continue;
        double dx[D], dv[D];
#pragma unroll
        for (int d = 0; d < D; ++d) dx[d] = xk[d] - S.x[d][i];
        const double r2 = dotD<D>(dx, dx);
        if (r2 > c.dpc_r2cut) continue;
        const double u = sqrt(r2) * c.dpc_l0inv;
        if (!(u < 1.0)) continue;
#pragma unroll
        for (int d = 0; d < D; ++d) dv[d] = vk[d] - S.v[d][i];
        const double chi = sqrt(wc2_w(u, c.dpc_nW) * c.dpc_whinv);
        const double vr = dotD<D>(dv, dx);
        double f;
        if (vr < 0.0) {
          f = -(u < c.dpc_kernlim ? 1.0 : chi) * (vr / (r2 + c.dpc_eta2));
        } else {
          const double Pb =
              chi * jl_max(jl_min(c.dpc_lambda * fabs(Pk + S.P1[i]), c.dpc_lambda * c.dpc_pmax), c.dpc_pmin);
          f = 2.0 * dt * Pb / ((rk + S.rho[i]) * (r2 + c.dpc_eta2));
        }
#pragma unroll
        for (int d = 0; d < D; ++d) sum[d] += f * dx[d];
      }
    }
    lanes_sum4<L>(sum, lane, group_mask<L>());
  }
  if (lane != 0) return;
  const double dt = sc->dt;
  S.Plast[k] = Pk;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    S.buf2[d][k] = sum[d];
    double nv = vk[d], nx = xk[d];
    if (ptk > 1) {
      nv = vk[d] + sum[d];
      nx = xk[d] + sum[d] * dt;
    }
    S.vo[d][k] = nv;
    S.xo[d][k] = nx;
    note_wild(S.wild, exponent(nv));
  }
}

// xsphcorr! + update_xsphcorr!  (:1757-1779, :1827-1838), stage-1 W
template <int D, int L>
__global__ void __launch_bounds__(STPB) k_xsph_rows(StepConst c, const Scal* __restrict__ sc, int64_t N, SArr<D> S) {
  if (*S.ovf) return;
  const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t k = gt / L;
  const int lane = (int)(gt % L);
  if (k >= N) return;
  double sum[4] = {0.0, 0.0, 0.0, 0.0};
  const int ptk = S.pt[k];
  if (ptk > 1) {
    double vk[D];
#pragma unroll
    for (int d = 0; d < D; ++d) vk[d] = S.v[d][k];
    const double rk = S.rho[k];
    const int64_t e1 = S.rs[k + 1];
    for (int64_t e = S.rs[k] + lane; e < e1; e += GATHER_U * L) {
      int32_t m[GATHER_U];
      int pt[GATHER_U];
      double w[GATHER_U], rm[GATHER_U], vm[GATHER_U][D];
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) {
        const bool in = e + j * L < e1;
        m[j] = in ? S.nbr[e + j * L] : (int32_t)k;
        w[j] = in ? S.We[e + j * L] : 0.0;
      }
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) {
        pt[j] = S.pt[m[j]];
        rm[j] = S.rho[m[j]];
#pragma unroll
        for (int d = 0; d < D; ++d) vm[j][d] = S.v[d][m[j]];
      }
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) {
        if (!(pt[j] > 1) || m[j] == k) continue;
        const double xs = w[j] * rcp_nr(rk + rm[j]);
#pragma unroll
        for (int d = 0; d < D; ++d) sum[d] += (vm[j][d] - vk[d]) * xs;
      }
    }
    // a sum of densities of 0 or infinity, where rcp_nr is NaN: again with the
    // division (rcp_any for every entry cost 0.6% of a call with surface
    // tension, 65k particles in 2-D)
    unsigned top = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) top = max(top, exponent(sum[d]));
    if (top == HI_INF) {
#pragma unroll
      for (int d = 0; d < D; ++d) sum[d] = 0.0;
#pragma unroll 1
      for (int64_t e = S.rs[k] + lane; e < e1; e += L) {
        const int32_t i = S.nbr[e];
        if (!(S.pt[i] > 1)) continue;
        const double xs = S.We[e] / (rk + S.rho[i]);
#pragma unroll
        for (int d = 0; d < D; ++d) sum[d] += (S.v[d][i] - vk[d]) * xs;
      }
    }
    lanes_sum4<L>(sum, lane, group_mask<L>());
  }
  if (lane != 0) return;
  const double dt = sc->dt;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const double u = sum[d] * (c.xsph_c * c.nW);
    S.buf2[d][k] = u;
    if (ptk > 1) S.x[d][k] = S.x[d][k] + u * dt;
  }
}

// cspmcorr!  (:1693-1719), stage-1 W; writes ρ to the other buffer
template <int D, int L>
__global__ void __launch_bounds__(STPB) k_cspm_rows(StepConst c, int64_t N, SArr<D> S) {
  if (*S.ovf) return;
  const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t k = gt / L;
  const int lane = (int)(gt % L);
  if (k >= N) return;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  const int ptk = S.pt[k];
  if (ptk > 0) {
    const int64_t e1 = S.rs[k + 1];
    for (int64_t e = S.rs[k] + lane; e < e1; e += GATHER_U * L) {
      int32_t m[GATHER_U];
      int pt[GATHER_U];
      double w[GATHER_U], rm[GATHER_U];
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) {
        const bool in = e + j * L < e1;
        m[j] = in ? S.nbr[e + j * L] : (int32_t)k;
        w[j] = in ? S.We[e + j * L] : 0.0;
      }
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) {
        pt[j] = S.pt[m[j]];
        rm[j] = S.rho[m[j]];
      }
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) {
        if (!(pt[j] > 0) || m[j] == k) continue;
        s[0] += w[j];
        s[1] += w[j] * rcp_any(rm[j]);
      }
    }
    lanes_sum4<L>(s, lane, group_mask<L>());
  }
  if (lane != 0) return;
  const double rk = S.rho[k];
  const double nr = s[0] / s[1];
  const double rv = isnan(nr) ? rk : nr;
  S.rhoo[k] = rv;
  const double Pk = eos(rv, c.gamma, c.rho0, c.P0, ptk), irk = 1.0 / rv;
  S.P1[k] = Pk;
  S.ir[k] = irk;
  note_wild(S.wild, max(exponent(rv), max(exponent(Pk), exponent(irk))));
  const double mw = c.m0 * c.nW;
  S.buf2[0][k] = s[0] * mw;
  S.buf2[1][k] = s[1] * mw;
  if (D == 3) S.buf2[2][k] = 0.0;
}

// The terms of a call's ∑W and ∑∇W by pair, into both rows' slots: (1 + 4u)
// (1 - u)^4 and Δx (1 - u)^3 for pairs of one side, zero for others.  FP64-bound,
// so once a pair; the row sums then read slots (rows that evaluated their
// entries, each pair twice: 3-D full physics, 23.5M pairs, a call 23.96 ms
// against 23.46; 3-D plain, 5.5M pairs, 7242 us against 7098; 2-D, 102k pairs,
// a call of one step 211 against 205).
// A pair at an infinite separation adds Δx 0 and one at a NaN NaN to ∑∇W (a
// particle that diverged within the step): the factor of its Δx.
__device__ __forceinline__ double no_pair(double r2) { return r2 == r2 ? 0.0 : NAN; }
constexpr int PS_TPB = 256;
template <int D>
__global__ void __launch_bounds__(PS_TPB) k_pair_sums(StepConst c, SArr<D> S, PairBuf B) {
  if (*S.ovf) return;
  const int64_t np = *B.npair, stride = (int64_t)gridDim.x * PS_TPB;
  for (int64_t u = (int64_t)blockIdx.x * PS_TPB + threadIdx.x; u < np; u += stride) {
    const int4 q = B.pq[u];  // (the last step's first stage has closed every mirror)
    double w = 0.0, g[3] = {0.0, 0.0, 0.0};
    if ((S.pt[q.x] > 0) == (S.pt[q.y] > 0)) {
      double dx[D];
#pragma unroll
      for (int d = 0; d < D; ++d) dx[d] = S.x[d][q.x] - S.x[d][q.y];
      const double r2 = dotD<D>(dx, dx);
      const bool r2pos = dbits(r2) != 0;
      const double t = r2pos ? fma(-sqrt_nr(r2), c.Hinv, 1.0) : 1.0;
      if ((unsigned long long)dbits(t) - 1ull < (unsigned long long)ONE_BITS) {
        const double t2 = t * t;
        w = fma(-4.0, t, 5.0) * (t2 * t2);
        const double t3 = r2pos ? t2 * t : NAN;  // the reference's d𝒲(0)/0
#pragma unroll
        for (int d = 0; d < D; ++d) g[d] = dx[d] * t3;
      } else if (exponent(r2) == HI_INF) {
#pragma unroll
        for (int d = 0; d < D; ++d) g[d] = dx[d] * no_pair(r2);
      }
    }
    put_slot(B.ce + q.z, w, g[0], g[1], g[2]);
    put_slot(B.ce + q.w, w, flip(g[0]), flip(g[1]), flip(g[2]));
  }
}

// post-batch sph∑W! + sph∑∇W!  (:139-156, :332-359).  The kernel's factors
// come out of the sums: ∑W = nW ∑ (1 + 4u)(1 - u)^4, ∑∇W = dWg ∑ Δx (1 - u)^3.
// With SCATTER (after a step) the terms are k_pair_sums's slots, and the lanes
// of a particle also write its state back to the original order, an array in
// turn each; without (no step in the call) the rows evaluate their entries.
template <int D, int L, bool SCATTER>
__global__ void __launch_bounds__(STPB) k_sums_rows(StepConst c, int64_t N, const int64_t* __restrict__ rs,
                                                    const int32_t* __restrict__ nbr, PostSums Q,
                                                    const int* __restrict__ ovf, StateIO<D> O, SArr<D> S,
                                                    const PairOut* ce) {
  if (*ovf) return;
  const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t k = gt / L;
  const int lane = (int)(gt % L);
  if (k >= N) return;
  const int32_t ik = Q.map ? Q.map[k] : (int32_t)k;
  double xk[D];
#pragma unroll
  for (int d = 0; d < D; ++d) xk[d] = Q.x[d][ik];
  const bool real = Q.pt[ik] > 0;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  const int64_t e1 = rs[k + 1];
  if constexpr (SCATTER) {
    for (int64_t e = rs[k] + lane; e < e1; e += 4 * L) {
      double v[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (e + j * L < e1) get_slot(ce + e + j * L, v[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (e + j * L < e1)
#pragma unroll
          for (int d = 0; d < 1 + D; ++d) s[d] += v[j][d];
    }
  }
  if constexpr (!SCATTER) {
    for (int64_t e = rs[k] + lane; e < e1; e += GATHER_U * L) {
      int32_t m[GATHER_U];
      int pt[GATHER_U];
      double xm[GATHER_U][D];
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) m[j] = e + j * L < e1 ? nbr[e + j * L] : -1;
      if (Q.map) {
#pragma unroll
        for (int j = 0; j < GATHER_U; ++j) m[j] = m[j] < 0 ? -1 : Q.map[m[j]];
      }
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) {
        const int32_t i = m[j] < 0 ? ik : m[j];
        pt[j] = Q.pt[i];
#pragma unroll
        for (int d = 0; d < D; ++d) xm[j][d] = Q.x[d][i];
      }
#pragma unroll
      for (int j = 0; j < GATHER_U; ++j) {
        if (m[j] < 0 || (pt[j] > 0) != real) continue;
        double dx[D];
#pragma unroll
        for (int d = 0; d < D; ++d) dx[d] = xk[d] - xm[j][d];
        const double r2 = dotD<D>(dx, dx);
        const bool r2pos = dbits(r2) != 0;
        const double u = r2pos ? sqrt_nr(r2) * c.Hinv : 0.0;
        if (!(u < 1.0)) {
          if (!(r2 < INFINITY)) {
#pragma unroll
            for (int d = 0; d < D; ++d) s[1 + d] += dx[d] * no_pair(r2);
          }
          continue;
        }
        const double t = 1.0 - u, t2 = t * t;
        s[0] += fma(4.0, u, 1.0) * (t2 * t2);
        const double t3 = r2pos ? t2 * t : NAN;  // the reference's d𝒲(0)/0
#pragma unroll
        for (int d = 0; d < D; ++d) s[1 + d] += dx[d] * t3;
      }
    }
  }
  lanes_sum4<L>(s, lane, group_mask<L>());
  const int32_t o = Q.orig[k];
  if constexpr (SCATTER) {
    if (lane == 0) {
      O.rho[o] = S.rho[k];
      O.rhoh[o] = S.rhoh[k];
      O.drho[o] = S.drho[k];
      O.P[o] = S.Plast[k];
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (lane == (1 + 2 * d) % L) {
        O.x[d][o] = xk[d];
        O.v[d][o] = S.v[d][k];
        O.vh[d][o] = S.vh[d][k];
      }
      if (lane == (2 + 2 * d) % L) {
        O.xh[d][o] = S.xh[d][k];
        O.cdx[d][o] = S.cdx[d][k];
        O.a[d][o] = S.a[d][k];
        O.buf2[d][o] = S.buf2[d][k];
      }
    }
  }
  if (lane != 0) return;
  Q.sumW[o] = s[0] * c.nW;
#pragma unroll
  for (int d = 0; d < D; ++d) Q.sg[d][o] = s[1 + d] * c.dWg;
}

template <int D, int STAGE, bool QUEUE>
static int pairA_grid(int* g) {
  // one block per SM (the kernel's registers leave room for one);
  // the occupancy query covers a build where two would fit
  static int grid = 0;
  if (grid == 0) {
    int dev = 0, sms = 0, per = 0;
    GC_CUDA(cudaGetDevice(&dev));
    GC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    GC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pairA<D, STAGE, QUEUE>, pa_tpb<QUEUE>(), 0));
    grid = sms * (per > 0 ? per : 1);
  }
  *g = grid;
  return GCSPH_OK;
}

template <int D, int STAGE>
static int run_pairA(cudaStream_t st, const StepConst& c, const SArr<D>& S, const PairBuf& B, int64_t pairs_est) {
  int g = 0, rc;
  if ((rc = pairA_grid<D, STAGE, false>(&g))) return rc;
  if (pairs_est <= (int64_t)g * pa_tpb<false>()) {  // about one chunk a warp
    k_pairA<D, STAGE, false><<<g, pa_tpb<false>(), 0, st>>>(c, S, B);
  } else {
    if ((rc = pairA_grid<D, STAGE, true>(&g))) return rc;
    k_pairA<D, STAGE, true><<<g, pa_tpb<true>(), 0, st>>>(c, S, B);
  }
  GC_LAUNCHED();
  return GCSPH_OK;
}

// pairs_est: about how many pairs the list holds (the count itself is on the
// device); it picks the form, both run any count
template <int D>
int launch_pairA(int stage, cudaStream_t st, const StepConst& c, const SArr<D>& S, const PairBuf& B,
                 int64_t pairs_est) {
  return stage == 1 ? run_pairA<D, 1>(st, c, S, B, pairs_est) : run_pairA<D, 2>(st, c, S, B, pairs_est);
}

template <int D>
int launch_pairB(int stage, int L, int64_t N, cudaStream_t st, const StepConst& c, Scal* sc, const SArr<D>& S,
                 const PairBuf& B, const NextBin* nb, const PosCopy* pc) {
  const int g = nblocks(N, 32);  // 32 particles per block, 32 L threads
  const NextBin nbv = nb ? *nb : NextBin{};
  const PosCopy pcv = pc ? *pc : PosCopy{};
#define GC_PAIRB(LL)                                                        \
  if (stage == 1)                                                          \
    k_pairB1<D, LL><<<g, 32 * LL, 0, st>>>(c, sc, N, S, B);                \
  else                                                                     \
    k_pairB2<D, LL><<<g, 32 * LL, 0, st>>>(c, sc, N, S, B, nbv, pcv);
  switch (L) {
    case 2: GC_PAIRB(2) break;
    case 4: GC_PAIRB(4) break;
    case 8: GC_PAIRB(8) break;
    case 16: GC_PAIRB(16) break;
    default: GC_PAIRB(32) break;
  }
#undef GC_PAIRB
  GC_LAUNCHED();
  return GCSPH_OK;
}

#define GC_ROWS(KER, ...)                                          \
  do {                                                             \
    const int g = nblocks(N * (int64_t)L, STPB);                   \
    switch (L) {                                                   \
      case 2: KER<D, 2><<<g, STPB, 0, st>>>(__VA_ARGS__); break;   \
      case 4: KER<D, 4><<<g, STPB, 0, st>>>(__VA_ARGS__); break;   \
      case 8: KER<D, 8><<<g, STPB, 0, st>>>(__VA_ARGS__); break;   \
      case 16: KER<D, 16><<<g, STPB, 0, st>>>(__VA_ARGS__); break; \
      default: KER<D, 32><<<g, STPB, 0, st>>>(__VA_ARGS__); break; \
    }                                                              \
    GC_LAUNCHED();                                                 \
    return GCSPH_OK;                                               \
  } while (0)

template <int D>
int launch_dpc(int L, int64_t N, cudaStream_t st, const StepConst& c, const Scal* sc, const SArr<D>& S,
               const PosCopy& pc) {
  GC_ROWS(k_dpc_rows, c, sc, N, S, pc);
}
template <int D>
int launch_xsph(int L, int64_t N, cudaStream_t st, const StepConst& c, const Scal* sc, const SArr<D>& S) {
  GC_ROWS(k_xsph_rows, c, sc, N, S);
}
template <int D>
int launch_cspm(int L, int64_t N, cudaStream_t st, const StepConst& c, const SArr<D>& S) {
  GC_ROWS(k_cspm_rows, c, N, S);
}
template <int D>
int launch_sums_post(int L, int64_t N, cudaStream_t st, const StepConst& c, const int64_t* rs, const int32_t* nbr,
                     const PostSums& Q, const int* ovf, bool scatter, const StateIO<D>& O, const SArr<D>& S,
                     const PairBuf& B, int64_t pairs_est) {
  const PairOut* ce = B.ce;
  if (scatter) {
    static int sms = 0;
    if (sms == 0) {
      int dev = 0;
      GC_CUDA(cudaGetDevice(&dev));
      GC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    }
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>(nblocks(pairs_est, PS_TPB), sms * 16));
    k_pair_sums<D><<<g, PS_TPB, 0, st>>>(c, S, B);
    GC_LAUNCHED();
  }
#define GC_SUMS(LL)                                                                                            \
  if (scatter)                                                                                                 \
    k_sums_rows<D, LL, true><<<nblocks(N * (int64_t)LL, STPB), STPB, 0, st>>>(c, N, rs, nbr, Q, ovf, O, S, ce); \
  else                                                                                                         \
    k_sums_rows<D, LL, false><<<nblocks(N * (int64_t)LL, STPB), STPB, 0, st>>>(c, N, rs, nbr, Q, ovf, O, S, ce);
  switch (L) {
    case 2: GC_SUMS(2) break;
    case 4: GC_SUMS(4) break;
    case 8: GC_SUMS(8) break;
    case 16: GC_SUMS(16) break;
    default: GC_SUMS(32) break;
  }
#undef GC_SUMS
  GC_LAUNCHED();
  return GCSPH_OK;
}
#undef GC_ROWS

#define GC_INST(D)                                                                                                \
  template int launch_dpc<D>(int, int64_t, cudaStream_t, const StepConst&, const Scal*, const SArr<D>&,          \
                             const PosCopy&);                                                                     \
  template int launch_xsph<D>(int, int64_t, cudaStream_t, const StepConst&, const Scal*, const SArr<D>&);         \
  template int launch_cspm<D>(int, int64_t, cudaStream_t, const StepConst&, const SArr<D>&);                      \
  template int launch_sums_post<D>(int, int64_t, cudaStream_t, const StepConst&, const int64_t*, const int32_t*,  \
                                   const PostSums&, const int*, bool, const StateIO<D>&, const SArr<D>&, const PairBuf&, int64_t);
GC_INST(2)
GC_INST(3)
#undef GC_INST
template int launch_pairA<2>(int, cudaStream_t, const StepConst&, const SArr<2>&, const PairBuf&, int64_t);
template int launch_pairA<3>(int, cudaStream_t, const StepConst&, const SArr<3>&, const PairBuf&, int64_t);
template int launch_pairB<2>(int, int, int64_t, cudaStream_t, const StepConst&, Scal*, const SArr<2>&,
                             const PairBuf&, const NextBin*, const PosCopy*);
template int launch_pairB<3>(int, int, int64_t, cudaStream_t, const StepConst&, Scal*, const SArr<3>&,
                             const PairBuf&, const NextBin*, const PosCopy*);

}  // namespace gcsph
