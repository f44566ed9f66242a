// celllist_upper.cu -- the cell list's own pair list (update! / partialupdate!
// and their emit): the pairs k < m alone, one thread per point.
//
// Each sorted point k has one sequence of candidates, m = k + 1 .. in its own
// x-row and then the rows of the half stencil that follow in key order (1 more
// row in 2-D, 4 more in 3-D).  A thread walks its point's candidates 32 at a
// time into a word of hit bits.  Sets of few candidates a point (UP_FEW words)
// keep the words; denser ones keep the neighbours themselves, expanded from
// each word as it is made.  The emit turns either into the caller's (min, max)
// list.  Ascending m is the order of both, so the list is the one a search that
// writes neighbours in turn would give.
//
// Why one thread per point: with a group of lanes per point, every candidate
// paid for a ballot, two popcounts and a scattered store besides its five
// floating-point instructions -- some 84 instructions per 32 candidates and
// point -- and the neighbour rows went through memory three times (staged,
// copied into a CSR, read back by the emit).  A thread that walks its own
// candidates needs about ten per candidate, and the lanes of a warp are points
// of the same or neighbouring cells, so their loads fall on the same few
// lines.  Measured (one GB300): search and emit of 200k uniform 2-D points (79
// pairs a point) 131 + 61 + 67 -> 71 + 43 us; of 333k uniform 3-D points (43 a
// point) 354 + 89 + 58 -> 108 + 49 us; of 4M uniform 3-D points (4.3 a point) 685 +
// 125 + 86 -> 202 + 100 us.
//
// Compiled without FMA contraction: r2_ref is the reference's expression.
#include <algorithm>
#include "celllist.cuh"

namespace gcsph {

static constexpr int UTPB = 256;
// Sets of up to this many words of candidates a point keep the words.  update!
// with words and with rows, us, at 1.2 / 1.8 / 2.2 / 3 / 4 words: 300k points in
// 2-D 149 149, 163 160, 184 174, 219 196, 271 209; 300k in 3-D 149 149, 152 149,
// 160 157, 177 173, 196 183; 2M in 3-D 356 409, 386 445, 432 475, 517 535, 680 606.
static constexpr double UP_FEW = 2.0;
// pairs collected per block of their emit (16 KB)
static constexpr int EMIT_STAGE = 2048;

// the FP32 prefilter copy, one vector per point
template <int D> struct PfVec;
template <> struct PfVec<2> { using T = float2; };
template <> struct PfVec<3> { using T = float4; };
template <int D>
__device__ __forceinline__ typename PfVec<D>::T pf_make(const float* v) {
  if constexpr (D == 2) return make_float2(v[0], v[1]);
  else return make_float4(v[0], v[1], v[2], 0.f);
}

template <int D>
constexpr int UP_GROUP = D == 2 ? 8 : 4;  // candidates tested at a time, and the vectors' padding

// one point's positions into cell order: FP64 copies, the FP32 prefilter
// vector and its bound (abs_hi; a NaN coordinate sends every candidate of the
// set to FP64)
template <int D>
__device__ __forceinline__ unsigned place_point(const double* xv, const Grid& g, int64_t k, double* const* xs,
                                              typename PfVec<D>::T* pf) {
  unsigned b = 0;
  float f[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    xs[d][k] = xv[d];
    const double v = xv[d] - g.offset[d];
    f[d] = (float)v;
    b = max(b, abs_hi(v));
  }
  pf[k] = pf_make<D>(f);
  return b;
}

struct Pos3 {
  const double* in[3];
  double* out[3];
};

// the rank of each point of the arrival lists among its cell's by original
// index, and its place in cell order at once
template <int D>
__global__ void __launch_bounds__(UTPB) k_rank_place(const PointRec* __restrict__ rec,
                                                     const int32_t* __restrict__ cellstart, int64_t N, Grid g,
                                                     int32_t* __restrict__ perm, int32_t* __restrict__ skey,
                                                     int32_t* __restrict__ orig, Pos3 P,
                                                     typename PfVec<D>::T* __restrict__ pf, unsigned long long* bmax,
                                                     float2* thr, unsigned* cnt) {
  const int64_t q = (int64_t)blockIdx.x * UTPB + threadIdx.x;
  unsigned b = 0;
  if (q < N) {
    const PointRec p = rec[q];
    const int32_t s = cellstart[p.key], e = cellstart[p.key + 1];
    int32_t r = 0;
#pragma unroll 4
    for (int32_t t = s; t < e; ++t) r += rec[t].i < p.i;
    const int64_t k = s + r;
    perm[k] = p.i;
    skey[k] = p.key;
    orig[k] = p.i;
    b = place_point<D>(p.x, g, k, P.out, pf);
  }
  atomic_max_hi(bmax, b);
  pf_thresholds_last_block<D>(bmax, g.dist2, thr, cnt);
}

// positions by a map (a radix-sorted binning, or stale cells with moved points)
template <int D>
__global__ void __launch_bounds__(UTPB) k_place(const int32_t* __restrict__ map, int64_t N, Grid g, Pos3 P,
                                                typename PfVec<D>::T* __restrict__ pf, unsigned long long* bmax,
                                                float2* thr, unsigned* cnt) {
  const int64_t k = (int64_t)blockIdx.x * UTPB + threadIdx.x;
  unsigned b = 0;
  if (k < N) {
    const int32_t i = map[k];
    double xv[D];
#pragma unroll
    for (int d = 0; d < D; ++d) xv[d] = P.in[d][i];
    b = place_point<D>(xv, g, k, P.out, pf);
  }
  atomic_max_hi(bmax, b);
  pf_thresholds_last_block<D>(bmax, g.dist2, thr, cnt);
}

// The candidate rows of point k, in key order: its own row from k + 1 on,
// then the stencil's later rows (empty outside the grid).  Row r holds the
// candidates c[r - 1] <= t < c[r] of the sequence, candidate t is the point
// t + dl[r].
template <int D>
struct UpRows {
  static constexpr int R = D == 2 ? 2 : 5;
  int32_t dl[R], c[R];
  __device__ __forceinline__ int32_t total() const { return c[R - 1]; }
  __device__ __forceinline__ int32_t at(int32_t t) const {
    int32_t d = dl[0];
#pragma unroll
    for (int r = 1; r < R; ++r)
      if (t >= c[r - 1]) d = dl[r];
    return t + d;
  }
};

template <int D>
__device__ __forceinline__ UpRows<D> up_rows(int64_t k, int32_t key, const int32_t* __restrict__ cellstart,
                                             const Grid& g) {
  const int nx = g.nc[0], ny = g.nc[1], nz = D == 3 ? g.nc[2] : 1;
  const int t = g.fx.quot(key);
  const int cx = key - t * nx;
  const int cz = D == 3 ? g.fy.quot(t) : 0;
  const int cy = t - cz * ny;
  const int xlo = cx > 0 ? cx - 1 : 0, xhi = cx < nx - 1 ? cx + 1 : nx - 1;
  constexpr int R = UpRows<D>::R;
  int32_t m0[R], m1[R];
  m0[0] = (int32_t)k + 1;
  m1[0] = cellstart[key - cx + xhi + 1];
#pragma unroll
  for (int r = 1; r < R; ++r) {
    const int dy = r == 1 ? 1 : r - 3, dz = r == 1 ? 0 : 1;
    const int y = cy + dy, z = cz + dz;
    m0[r] = m1[r] = 0;
    if (y >= 0 && y < ny && z < nz) {
      const int base = nx * (y + ny * z);  // fewer than 2^31 cells
      m0[r] = cellstart[base + xlo];
      m1[r] = cellstart[base + xhi + 1];
    }
  }
  UpRows<D> U;
  int32_t c = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    U.dl[r] = m0[r] - c;
    c += m1[r] - m0[r];
    U.c[r] = c;
  }
  return U;
}

// the FP32 squared distance (any rounding of it lies inside the band)
template <int D>
__device__ __forceinline__ float r2_pf(const typename PfVec<D>::T& a, const typename PfVec<D>::T& b) {
  const float d0 = a.x - b.x, d1 = a.y - b.y;
  float r2 = fmaf(d1, d1, d0 * d0);
  if constexpr (D == 3) {
    const float d2 = a.z - b.z;
    r2 = fmaf(d2, d2, r2);
  }
  return r2;
}

// the reference's FP64 test of a candidate inside the band
template <int D>
__device__ __forceinline__ bool hit_exact(int64_t k, int32_t m, double* const* xs, double dist2) {
  return r2_ref<D>(xs[0][k], xs[1][k], D == 3 ? xs[2][k] : 0.0, xs[0][m], xs[1][m], D == 3 ? xs[2][m] : 0.0) < dist2;
}

// One thread walks all candidates of point k: chunk(m, n, in) gets the hit bits
// of the n <= 32 candidates from m on, in order.  UP_GROUP candidates at a time:
// eight in 2-D, four in 3-D, whose rows are short (8 there: 219 -> 230 us at 4M
// points; 4 in 2-D: 37 -> 41 us at 200k).  The vectors past the last point that
// a group may read are padding (their bits are cut off).
template <int D, class F>
__device__ __forceinline__ void up_walk(int64_t k, const UpRows<D>& U, const typename PfVec<D>::T* __restrict__ pf,
                                        double* const* xs, float2 tt, double dist2, F chunk) {
  constexpr int G = UP_GROUP<D>;
  const typename PfVec<D>::T a = pf[k];
#pragma unroll
  for (int r = 0; r < UpRows<D>::R; ++r) {
    const int32_t m1 = U.c[r] + U.dl[r];
    for (int32_t m = (r ? U.c[r ? r - 1 : 0] : 0) + U.dl[r]; m < m1; m += 32) {
      const int n = min(32, m1 - m);
      unsigned in = 0, ok = 0;  // surely in; not surely out
      for (int j = 0; j < n; j += G) {
        unsigned ig = 0, og = 0;
#pragma unroll
        for (int q = 0; q < G; ++q) {
          const float r2 = r2_pf<D>(a, pf[m + j + q]);
          if (r2 < tt.x) ig |= 1u << q;
          if (!(r2 > tt.y)) og |= 1u << q;
        }
        in |= ig << j;
        ok |= og << j;
      }
      const unsigned cut = n == 32 ? 0xffffffffu : (1u << n) - 1u;
      in &= cut;
      unsigned band = ok & cut & ~in;
      while (band) {
        const int b = __ffs(band) - 1;
        band &= band - 1;
        if (hit_exact<D>(k, m + b, xs, dist2)) in |= 1u << b;
      }
      chunk(m, n, in);
    }
  }
}

// Count pass: what each point keeps (ROWS: its neighbours, else its words; W of
// either, point-major), its offset among the pairs of its block, the blocks'
// totals and the candidate statistics; the last block of a grid of up to
// SCAN_FOLD_MAX blocks scans the totals into the blocks' starts
// (base[gridDim.x] is the total).
template <int D, bool ROWS>
__global__ void __launch_bounds__(UTPB, D == 2 ? 4 : 5) k_up_count(
    const typename PfVec<D>::T* __restrict__ pf, Pos3 P, const float2* __restrict__ thr,
    const int32_t* __restrict__ skey, const int32_t* __restrict__ cellstart, int64_t N, Grid g,
    unsigned* __restrict__ kept, int W, int32_t* __restrict__ loc, int32_t* __restrict__ total,
    int64_t* __restrict__ base, UpStat* stat, unsigned* fold_cnt) {
  const int64_t k = (int64_t)blockIdx.x * UTPB + threadIdx.x;
  int32_t cnt = 0, nw = 0;
  if (k < N) {
    const UpRows<D> U = up_rows<D>(k, skey[k], cellstart, g);
    nw = (U.total() + 31) >> 5;
    unsigned* kp = kept + k * W;
    if constexpr (ROWS) {
      // four neighbours to a store (W is a multiple of four)
      int4 v = make_int4(0, 0, 0, 0);
      up_walk<D>(k, U, pf, P.out, *thr, g.dist2, [&](int32_t m, int, unsigned in) {
        while (in) {
          const int b = __ffs(in) - 1;
          in &= in - 1;
          v = make_int4(v.y, v.z, v.w, m + b);
          ++cnt;
          if ((cnt & 3) == 0 && cnt <= W) *reinterpret_cast<int4*>(kp + cnt - 4) = v;
        }
      });
      const int left = cnt & 3;
      if (cnt < W) {
        unsigned* e = kp + (cnt - left);
        if (left == 3) e[0] = v.y;
        if (left >= 2) e[left - 2] = v.z;
        if (left >= 1) e[left - 1] = v.w;
      }
    } else {
      unsigned long long acc = 0;
      int fill = 0, w = 0;
      up_walk<D>(k, U, pf, P.out, *thr, g.dist2, [&](int32_t, int n, unsigned in) {
        cnt += __popc(in);
        acc |= (unsigned long long)in << fill;
        fill += n;
        if (fill >= 32) {
          if (w < W) kp[w] = (unsigned)acc;
          ++w;
          acc >>= 32;
          fill -= 32;
        }
      });
      if (fill > 0 && w < W) kp[w] = (unsigned)acc;
    }
  }
  // the block's exclusive scan of the counts; the sum of the words, and the
  // most of what a point keeps
  __shared__ int32_t s_c[UTPB / 32], s_s[UTPB / 32], s_m[UTPB / 32];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  int32_t inc = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  const int32_t ws = __reduce_add_sync(0xffffffffu, nw), wm = __reduce_max_sync(0xffffffffu, ROWS ? cnt : nw);
  if (lane == 31) {
    s_c[wp] = inc;
    s_s[wp] = ws;
    s_m[wp] = wm;
  }
  __syncthreads();
  int32_t before = 0, all = 0, sum = 0, mx = 0;
#pragma unroll
  for (int v = 0; v < UTPB / 32; ++v) {
    if (v < wp) before += s_c[v];
    all += s_c[v];
    sum += s_s[v];
    mx = max(mx, s_m[v]);
  }
  if (k < N) loc[k] = before + inc - cnt;
  if (threadIdx.x == 0) {
    total[blockIdx.x] = all;
    if (blockIdx.x % UP_SAMPLE == 0) atomicAdd(&stat->words, (unsigned long long)sum);
    if (mx > *(volatile int*)&stat->most) atomicMax(&stat->most, mx);
  }
  if (fold_cnt && last_block_of_grid(fold_cnt)) block_exclusive_scan<int64_t>(total, base, gridDim.x);
}

// (min, max) of a pair's 1-based original indices, and its store
__device__ __forceinline__ int2 make_pair1(int32_t ok, int32_t om) {
  return make_int2(min(ok, om), max(ok, om));
}
__device__ __forceinline__ void store_pair(int32_t* pairs, int64_t pos, int2 v, bool aligned) {
  if (aligned) {
    reinterpret_cast<int2*>(pairs)[pos] = v;
  } else {
    pairs[2 * pos] = v.x;
    pairs[2 * pos + 1] = v.y;
  }
}

// pairs of point k: those of its block's list from loc[k] on
__device__ __forceinline__ int32_t up_pairs(int64_t k, int64_t N, const int32_t* __restrict__ loc,
                                            const int32_t* __restrict__ total) {
  const int64_t kn = k + 1;
  return (kn < N && kn % UTPB != 0 ? loc[kn] : total[k / UTPB]) - loc[k];
}

// Emit from words, one thread per point: a block's pairs are one run of the
// list, so they are collected in shared memory and stored as such.  A point
// with more words than are kept is searched again.
template <int D>
__global__ void __launch_bounds__(UTPB, 6) k_up_emit_words(
    const typename PfVec<D>::T* __restrict__ pf, Pos3 P, const float2* __restrict__ thr,
    const int32_t* __restrict__ skey, const int32_t* __restrict__ cellstart, const int32_t* __restrict__ orig,
    int64_t N, Grid g, const unsigned* __restrict__ kept, int W, const int32_t* __restrict__ loc,
    const int32_t* __restrict__ total, const int64_t* __restrict__ base, int64_t cap, int32_t* __restrict__ pairs,
    bool aligned) {
  __shared__ int2 s_p[EMIT_STAGE];
  const int64_t k = (int64_t)blockIdx.x * UTPB + threadIdx.x;
  const int64_t b0 = base[blockIdx.x];
  const int32_t all = total[blockIdx.x];
  const bool staged = all <= EMIT_STAGE;
  if (k < N) {
    const UpRows<D> U = up_rows<D>(k, skey[k], cellstart, g);
    const int nw = (U.total() + 31) >> 5;
    const int32_t ok = orig[k] + 1;
    int32_t at = loc[k];
    auto pair = [&](int32_t m) {
      const int2 v = make_pair1(ok, orig[m] + 1);
      if (staged) s_p[at] = v;
      else if (b0 + at < cap) store_pair(pairs, b0 + at, v, aligned);
      ++at;
    };
    if (nw <= W) {
      for (int w = 0; w < nw; ++w) {
        unsigned word = kept[k * W + w];
        while (word) {
          pair(U.at(w * 32 + __ffs(word) - 1));
          word &= word - 1;
        }
      }
    } else {
      up_walk<D>(k, U, pf, P.out, *thr, g.dist2, [&](int32_t m, int, unsigned in) {
        while (in) {
          pair(m + __ffs(in) - 1);
          in &= in - 1;
        }
      });
    }
  }
  if (!staged) return;  // uniform over the block
  __syncthreads();
  for (int32_t i = threadIdx.x; i < all; i += UTPB)
    if (b0 + i < cap) store_pair(pairs, b0 + i, s_p[i], aligned);
}

// Emit from neighbour rows, L lanes per point, four entries of each in flight
// (at one the pass waits for its loads).  A row that outgrew its W entries is
// searched again by the group, L candidates at a time.
template <int D, int L>
__global__ void __launch_bounds__(UTPB) k_up_emit_rows(
    const typename PfVec<D>::T* __restrict__ pf, Pos3 P, const float2* __restrict__ thr,
    const int32_t* __restrict__ skey, const int32_t* __restrict__ cellstart, const int32_t* __restrict__ orig,
    int64_t N, Grid g, const unsigned* __restrict__ kept, int W, const int32_t* __restrict__ loc,
    const int32_t* __restrict__ total, const int64_t* __restrict__ base, int64_t cap, int32_t* __restrict__ pairs,
    bool aligned) {
  const int64_t gt = (int64_t)blockIdx.x * UTPB + threadIdx.x;
  const int64_t k = gt / L;
  const int lane = (int)(gt % L);
  if (k >= N) return;  // whole groups leave together
  const int32_t n = up_pairs(k, N, loc, total);
  const int32_t ok = orig[k] + 1;
  const int64_t pos = base[k / UTPB] + loc[k];
  int32_t* out = pairs + 2 * pos;
  const int32_t lim = (int32_t)max((int64_t)0, min(cap - pos, (int64_t)n));  // of this point's pairs, those that fit
  if (n <= W) {
    const int32_t* row = reinterpret_cast<const int32_t*>(kept) + k * W;
    for (int32_t t = lane; t < lim; t += 4 * L) {
      int32_t om[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) om[j] = t + j * L < lim ? row[t + j * L] : (int32_t)k;
#pragma unroll
      for (int j = 0; j < 4; ++j) om[j] = orig[om[j]] + 1;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (t + j * L < lim) store_pair(out, t + j * L, make_pair1(ok, om[j]), aligned);
    }
    return;
  }
  const unsigned gbase = threadIdx.x & 31u & ~(unsigned)(L - 1);
  const unsigned gm = L == 32 ? 0xffffffffu : ((1u << L) - 1u) << gbase;
  const UpRows<D> U = up_rows<D>(k, skey[k], cellstart, g);
  const int32_t tot = U.total();
  const typename PfVec<D>::T a = pf[k];
  int32_t off = 0;
  for (int32_t tb = 0; tb < tot; tb += L) {
    const int32_t t = tb + lane;
    int32_t m = 0;
    bool hit = false;
    if (t < tot) {
      m = U.at(t);
      const float r2 = r2_pf<D>(a, pf[m]);
      hit = r2 < thr->x || (!(r2 > thr->y) && hit_exact<D>(k, m, P.out, g.dist2));
    }
    const unsigned bal = (__ballot_sync(gm, hit) >> gbase) & (L == 32 ? 0xffffffffu : (1u << L) - 1u);
    const int32_t at = off + __popc(bal & ((1u << lane) - 1u));
    if (hit && at < lim) store_pair(out, at, make_pair1(ok, orig[m] + 1), aligned);
    off += __popc(bal);
  }
}

// ---------------------------------------------------------------------------
// The step's rows (both directions), one thread per point: k_pairs32's MODE 2
// -- the two counts, and the row staged ascending at stg[k * S ..] -- for sets
// large enough to fill the GPU with a thread each.  The prefilter's copies are
// the step's (one array per dimension, a group of padding past the last point).
// ---------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(UTPB, 4) k_full_count(
    const float* __restrict__ f0, const float* __restrict__ f1, const float* __restrict__ f2, Pos3 P,
    const float2* __restrict__ thr, const int32_t* __restrict__ skey, const int32_t* __restrict__ cellstart, int64_t N,
    Grid g, int32_t* __restrict__ cnt_full, int32_t* __restrict__ cnt_up, int32_t* __restrict__ stg, int S) {
  const int64_t k64 = (int64_t)blockIdx.x * UTPB + threadIdx.x;
  if (k64 >= N) return;
  const int32_t k = (int32_t)k64;
  constexpr int NR = D == 2 ? 3 : 9, G = 8;
  const int nx = g.nc[0], ny = g.nc[1], nz = D == 3 ? g.nc[2] : 1;
  const int32_t key = skey[k];
  const int t = g.fx.quot(key);
  const int cx = key - t * nx;
  const int cz = D == 3 ? g.fy.quot(t) : 0;
  const int cy = t - cz * ny;
  const int xlo = cx > 0 ? cx - 1 : 0, xhi = cx < nx - 1 ? cx + 1 : nx - 1;
  auto range = [&](int r, int32_t& a, int32_t& b) {
    const int y = cy + r % 3 - 1, z = cz + (D == 3 ? r / 3 - 1 : 0);
    a = b = 0;
    if (y >= 0 && y < ny && z >= 0 && z < nz) {
      const int base = nx * (y + ny * z);
      a = cellstart[base + xlo];
      b = cellstart[base + xhi + 1];
    }
  };
  const float2 tt = *thr;
  const float ax = f0[k], ay = f1[k], az = D == 3 ? f2[k] : 0.f;
  int32_t* row = stg + k64 * S;
  int32_t cnt = 0, up = 0;
  int4 v = make_int4(0, 0, 0, 0);
  int32_t m0, m1;
  range(0, m0, m1);
#pragma unroll 1
  for (int r = 0; r < NR; ++r) {
    int32_t a = m0;
    const int32_t b = m1;
    if (r + 1 < NR) range(r + 1, m0, m1);  // the next row's range, a row ahead
    for (; a < b; a += 32) {
      const int n = min(32, b - a);
      unsigned in = 0, ok = 0;  // surely in; not surely out
      for (int j = 0; j < n; j += G) {
        unsigned ig = 0, og = 0;
#pragma unroll
        for (int q = 0; q < G; ++q) {
          const int32_t m = a + j + q;
          const float d0 = ax - f0[m], d1 = ay - f1[m];
          float r2 = fmaf(d1, d1, d0 * d0);
          if (D == 3) {
            const float d2 = az - f2[m];
            r2 = fmaf(d2, d2, r2);
          }
          if (r2 < tt.x) ig |= 1u << q;
          if (!(r2 > tt.y)) og |= 1u << q;
        }
        in |= ig << j;
        ok |= og << j;
      }
      unsigned cut = n == 32 ? 0xffffffffu : (1u << n) - 1u;
      if (k >= a && k < a + n) cut &= ~(1u << (k - a));
      in &= cut;
      unsigned band = ok & cut & ~in;
      while (band) {
        const int e = __ffs(band) - 1;
        band &= band - 1;
        if (hit_exact<D>(k, a + e, P.out, g.dist2)) in |= 1u << e;
      }
      // the bits above k: all of a chunk past k, none of one before it
      up += __popc(a > k ? in : (a + 31 <= k ? 0u : in & (0xfffffffeu << (k - a))));
      while (in) {
        const int e = __ffs(in) - 1;
        in &= in - 1;
        v = make_int4(v.y, v.z, v.w, a + e);
        ++cnt;
        if ((cnt & 3) == 0 && cnt <= S) *reinterpret_cast<int4*>(row + cnt - 4) = v;
      }
    }
  }
  const int left = cnt & 3;
  if (cnt < S) {  // S is a multiple of four
    int32_t* e = row + (cnt - left);
    if (left == 3) e[0] = v.y;
    if (left >= 2) e[left - 2] = v.z;
    if (left >= 1) e[left - 1] = v.w;
  }
  cnt_full[k] = cnt;
  cnt_up[k] = up;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
template <int D>
static Pos3 pos3(const double* const* in, double* const* out) {
  Pos3 P{};
  for (int d = 0; d < D; ++d) {
    P.in[d] = in ? in[d] : nullptr;
    P.out[d] = out[d];
  }
  return P;
}

// A width: three times the mean, and in dense sets 256 past it, so that what is
// kept takes no more memory than the neighbours of all points in one array
// and a staged row of 256 each.
static double kept_room(double mean) { return std::min(3.0 * mean + 16.0, mean + 256.0); }
static int whole4(double w) { return ((int)w + 3) / 4 * 4; }

// The first search's form and width, from the grid-wide density: rows where a
// point has more than UP_FEW words of candidates (half a word of each point's
// is padding), as wide as kept_room allows for the pairs that the density gives
// a dist-ball.  A point at its cell's near edge has up to 2.7 times the mean of
// a uniform set, and a guess that one point outgrows costs a second search and
// another allocation (130 us of a small list's construction).
static void first_width(CellCore& C) {
  const double cand = 0.5 * C.candidates_per_point();
  C.up_rows = cand + 16.0 > 32.0 * UP_FEW;
  double pairs = cand * (C.D == 2 ? GCSPH_PI64 / 9.0 : 4.0 * GCSPH_PI64 / 81.0);
  for (int d = 0; d < C.D; ++d) pairs *= C.dist / C.cs[d];
  C.up_w = whole4(std::min(C.up_rows ? kept_room(pairs) : cand / 16.0 + 8.0, 4096.0));
}

size_t CellCore::kept_bytes() const {
  return (size_t)N * std::max(sizeof(unsigned) * (size_t)up_w, sizeof(PointRec));
}

// bytes of the search's buffers (cut from the cell list's allocation)
void CellCore::upper_sizes(size_t* upf_b, size_t* uptot_b, size_t* upbase_b, size_t* upstat_b, size_t* upkept_b) {
  const size_t nb = (size_t)nblocks(N, UTPB), n = (size_t)N;
  // (a group of padding, which a walk may read and cut off)
  *upf_b = D == 2 ? sizeof(PfVec<2>::T) * (n + UP_GROUP<2>) : sizeof(PfVec<3>::T) * (n + UP_GROUP<3>);
  *uptot_b = sizeof(int32_t) * (nb + 4);
  *upbase_b = sizeof(int64_t) * (nb + 1);
  *upstat_b = sizeof(UpStat);
  first_width(*this);
  *upkept_b = kept_bytes();
}

template <int D>
static int build_upper_impl(CellCore& C, const double* const* xin, double* const* xs, bool rebin) {
  using V = typename PfVec<D>::T;
  cudaStream_t st = C.st;
  const int64_t N = C.N;
  const int nb = nblocks(N, UTPB);
  int rc;
  if ((rc = C.ensure_pf_scalars())) return rc;
  V* pf = C.upf.as<V>();
  const Pos3 P = pos3<D>(xin, xs);
  unsigned long long* bm = C.pfmax.as<unsigned long long>();
  float2* thr = C.pfthr.as<float2>();
  unsigned* cnt = C.pfcnt.as<unsigned>();
  bool deferred = false;
  if (C.up_w == 0) first_width(C);
  if ((rc = C.upkept.ensure(C.kept_bytes(), st))) {
    C.up_w = 0;  // the next build guesses anew
    return rc;
  }
  // the records of the binning's arrival lists lie where the search that
  // follows keeps its words or rows
  if (rebin) {
    if ((rc = C.sort(xin, nullptr, true, &deferred, false, C.upkept.as<PointRec>()))) return rc;
  }
  if (!C.sorted && !deferred) return fail(GCSPH_ESTATE, "pair build before binning");
  timer_begin(T_SORT, st);
  if (deferred) {
    k_rank_place<D><<<nb, UTPB, 0, st>>>(C.upkept.as<PointRec>(), C.cellstart.as<int32_t>(), N, C.g,
                                         C.perm.as<int32_t>(), C.skey.as<int32_t>(), C.orig_b.as<int32_t>(), P, pf,
                                         bm, thr, cnt);
    GC_LAUNCHED();
    C.sort_done();
  } else {
    // stale cells: the points are the caller's, by original index
    k_place<D><<<nb, UTPB, 0, st>>>(rebin ? C.perm.as<int32_t>() : C.orig.as<int32_t>(), N, C.g, P, pf, bm, thr, cnt);
    GC_LAUNCHED();
  }
  timer_end(T_SORT, st);
  timer_begin(T_PAIRS, st);
  // What a point keeps: as much as the last search's fullest point needed and
  // a quarter more, up to kept_room (a crowded cell's points are searched again
  // in the emit).  A search that finds its points in need of more, or of the
  // other form, is run again; the width stays while the form does.
  const bool fold = nb <= SCAN_FOLD_MAX;
  for (;;) {
    if ((rc = C.upkept.ensure(C.kept_bytes(), st))) {
      C.up_w = 0;  // the next build guesses anew
      return rc;
    }
    GC_CUDA(cudaMemsetAsync(C.upstat.p, 0, sizeof(UpStat), st));
    const auto count = C.up_rows ? k_up_count<D, true> : k_up_count<D, false>;
    count<<<nb, UTPB, 0, st>>>(pf, P, thr, C.skey.as<int32_t>(), C.cellstart.as<int32_t>(), N, C.g,
                               C.upkept.as<unsigned>(), C.up_w, C.cnt_up.as<int32_t>(), C.uptot.as<int32_t>(),
                               C.upbase.as<int64_t>(), C.upstat.as<UpStat>(),
                               fold ? C.foldcnt.as<unsigned>() + 1 : nullptr);
    GC_LAUNCHED();
    if (!fold && (rc = exclusive_scan_i32_to_i64(C.uptot.as<int32_t>(), C.upbase.as<int64_t>(), nb,
                                                 C.scratch.as<int64_t>(), st)))
      return rc;
    GC_CUDA(cudaMemcpyAsync(C.pin, C.upbase.as<int64_t>() + nb, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    GC_CUDA(cudaMemcpyAsync(C.pin + 2, C.upstat.p, sizeof(UpStat), cudaMemcpyDeviceToHost, st));
    GC_CUDA(cudaStreamSynchronize(st));
    UpStat s;
    memcpy(&s, C.pin + 2, sizeof(s));
    int64_t sampled = (int64_t)((nb + UP_SAMPLE - 1) / UP_SAMPLE) * UTPB;
    if (sampled > N) sampled = N;
    const double words = (double)s.words / (double)sampled;
    const double mean = C.up_rows ? (double)C.pin[0] / (double)N : words;
    // (a set near the line between the forms stays with the one it has)
    if (C.up_rows ? words < 0.8 * UP_FEW : words > UP_FEW) {
      C.up_rows = !C.up_rows;
      // the other form's need: at a first guess its mean
      const double other = C.up_rows ? (double)C.pin[0] / (double)N : words;
      C.up_w = whole4(std::min(1.5 * other + 8.0, kept_room(other)));
      continue;
    }
    const double bound = kept_room(mean), most = std::min((double)s.most, bound);
    if (whole4(most) <= C.up_w) break;
    C.up_w = whole4(std::min(1.25 * most, bound));
  }
  timer_end(T_PAIRS, st);
  timer_collect();
  C.nup = C.pin[0];
  C.nfull = C.nup;
  C.nfull_est = 2 * C.nup;
  C.built = true;
  C.up_valid = true;
  C.rows_upper = true;
  return GCSPH_OK;
}

template <int D>
static int emit_upper_impl(CellCore& C, double* const* xs, int32_t* pairs, int64_t cap) {
  using V = typename PfVec<D>::T;
  cudaStream_t st = C.st;
  const int64_t N = C.N;
  const Pos3 P = pos3<D>(nullptr, xs);
  const bool aligned = ((uintptr_t)pairs & 7u) == 0;
#define UP_EMIT(KER, T)                                                                                            \
  KER<<<nblocks(T, UTPB), UTPB, 0, st>>>(C.upf.as<V>(), P, C.pfthr.as<float2>(), C.skey.as<int32_t>(),             \
                                         C.cellstart.as<int32_t>(), C.orig.as<int32_t>(), N, C.g,                  \
                                         C.upkept.as<unsigned>(), C.up_w, C.cnt_up.as<int32_t>(),                  \
                                         C.uptot.as<int32_t>(), C.upbase.as<int64_t>(), cap, pairs, aligned)
  if (!C.up_rows) {
    UP_EMIT((k_up_emit_words<D>), N);
  } else {
    // lanes per point: about four or five of its pairs each
    const double mean = (double)C.nup / (double)N;
    if (mean <= 24.0) UP_EMIT((k_up_emit_rows<D, 4>), N * 4);
    else if (mean <= 48.0) UP_EMIT((k_up_emit_rows<D, 8>), N * 8);
    else if (mean <= 96.0) UP_EMIT((k_up_emit_rows<D, 16>), N * 16);
    else UP_EMIT((k_up_emit_rows<D, 32>), N * 32);
  }
#undef UP_EMIT
  GC_LAUNCHED();
  return GCSPH_OK;
}

int CellCore::count_rows(const double* const* xs, int32_t* stg, int S) {
  Pos3 P{};
  for (int d = 0; d < D; ++d) P.out[d] = const_cast<double*>(xs[d]);
  const int nb = nblocks(N, UTPB);
  const float* f0 = pf[0].as<float>();
  const float* f1 = pf[1].as<float>();
  if (D == 2)
    k_full_count<2><<<nb, UTPB, 0, st>>>(f0, f1, f0, P, pfthr.as<float2>(), skey.as<int32_t>(), cellstart.as<int32_t>(),
                                         N, g, cnt_full.as<int32_t>(), cnt_up.as<int32_t>(), stg, S);
  else
    k_full_count<3><<<nb, UTPB, 0, st>>>(f0, f1, pf[2].as<float>(), P, pfthr.as<float2>(), skey.as<int32_t>(),
                                         cellstart.as<int32_t>(), N, g, cnt_full.as<int32_t>(), cnt_up.as<int32_t>(),
                                         stg, S);
  return GCSPH_OK;  // the caller counts and checks the launch
}

int CellCore::build_upper(const double* const* xin, double* const* xs, bool rebin) {
  list_gone();
  up_xs[0] = xs[0];
  up_xs[1] = xs[1];
  up_xs[2] = D == 3 ? xs[2] : nullptr;
  return D == 2 ? build_upper_impl<2>(*this, xin, xs, rebin) : build_upper_impl<3>(*this, xin, xs, rebin);
}

int CellCore::emit_upper(int32_t* pairs, int64_t cap) {
  return D == 2 ? emit_upper_impl<2>(*this, up_xs, pairs, cap) : emit_upper_impl<3>(*this, up_xs, pairs, cap);
}

}  // namespace gcsph
