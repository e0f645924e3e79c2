// fues.cu -- FUES upper envelope of DC-EGM candidate rows (kernel c, part 2).
//
// Restates the Fast Upper-Envelope Scan (Dobrescu & Shanker 2022) with the
// reference's rules (src/_lcm/egm/upper_envelope/fues.py:151-1189):
//   1. sort each row by (grid asc, value desc, policy desc), NaN grid last,
//      ties by input position (a stable lexsort);
//   2. reduce every run of equal grid values to its maximisers, keeping one
//      copy per exogenous savings source;
//   3. scan the sorted row keeping the last two envelope points (k, j); drop a
//      candidate below j on the same segment, one with falling savings and a
//      secant below the previous gradient, or one below the continuation of
//      j's segment; insert segment crossings twice (left / right policy);
//      "same segment" means |d(R - c)/dR| <= jump_thresh.
//
// GPU mapping: one CTA per row.  The CTA sorts an index array in shared
// memory (bitonic), gathers the sorted row into the workspace, reduces the
// coincident groups in parallel, and then warp 0 runs the scan: the scan
// state is held redundantly by all 32 lanes, and each exhaustive look-ahead
// for the next same-segment candidate inspects 32 candidates per step with
// a warp ballot.  Lane 0 writes the emissions.

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>

#include "../../include/lcmx.h"

namespace {

constexpr int kBlock = 256;
constexpr int kMaxSort = 8192;  // largest row the shared-memory sort handles

__device__ __forceinline__ bool isnan_(double x) { return x != x; }

__device__ __forceinline__ double slope(double xa, double ya, double xb, double yb) {
  const double dx = xb - xa;
  return dx == 0.0 ? 0.0 : (yb - ya) / dx;
}

// different segments iff the implied savings (R - c) jump
__device__ __forceinline__ bool policy_jump(double ga, double pa, double gb, double pb, double thr,
                                            bool use_sav, double sa, double sb) {
  const double ia = ga - pa, ib = gb - pb;
  if (ga == gb) return use_sav ? (sa != sb) : (ia != ib);
  return fabs(slope(ga, ia, gb, ib)) > thr;
}

__device__ __forceinline__ void intersect(double xa, double ya, double sa, double xb, double yb, double sb,
                                          double& x, double& y) {
  const double den = sa - sb;
  if (den == 0.0) {
    x = __longlong_as_double(0x7ff8000000000000LL);
    y = ya;
    return;
  }
  x = (yb - ya + sa * xa - sb * xb) / den;
  y = ya + sa * (x - xa);
}

struct Key {
  double g, v, p;
  int i;
};

__device__ __forceinline__ Key load_key(const double* g, const double* v, const double* p, int i, int n) {
  Key k;
  k.i = i;
  if (i >= n) {
    k.g = __longlong_as_double(0x7ff0000000000000LL);  // padding sorts last
    k.v = -k.g;
    k.p = -k.g;
    k.i = 0x7fffffff;
    return k;
  }
  const double gi = g[i], vi = v[i], pi = p[i];
  k.g = isnan_(gi) ? __longlong_as_double(0x7ff0000000000000LL) : gi;
  k.v = isnan_(vi) ? -__longlong_as_double(0x7ff0000000000000LL) : vi;
  k.p = isnan_(pi) ? -__longlong_as_double(0x7ff0000000000000LL) : pi;
  return k;
}

// a before b ?
__device__ __forceinline__ bool key_less(const Key& a, const Key& b) {
  if (a.g != b.g) return a.g < b.g;
  if (a.v != b.v) return a.v > b.v;
  if (a.p != b.p) return a.p > b.p;
  return a.i < b.i;
}

// first same-segment candidate from idx in direction dir among the `window`
// positions idx + dir, ..., idx + dir * window (warp-cooperative)
__device__ __forceinline__ bool find_same_segment(const double* g, const double* p, const double* v, int n,
                                                  double ag, double ap, int idx, int dir, double thr, int window,
                                                  double& fg, double& fp, double& fv) {
  const int lane = threadIdx.x & 31;
  for (int base = idx + dir;; base += 32 * dir) {
    if (dir > 0 ? base >= n : base < 0) break;
    if ((base - idx) * dir > window) break;
    const int k = base + dir * lane;
    bool ok = false;
    double gk = 0.0, pk = 0.0, vk = 0.0;
    if (k >= 0 && k < n && (k - idx) * dir <= window) {
      gk = g[k];
      pk = p[k];
      vk = v[k];
      ok = !isnan_(gk) && !isnan_(vk) && !policy_jump(ag, ap, gk, pk, thr, false, 0.0, 0.0);
    }
    const unsigned m = __ballot_sync(0xffffffffu, ok);
    if (m) {
      const int src = __ffs(m) - 1;  // nearest candidate
      fg = __shfl_sync(0xffffffffu, gk, src);
      fp = __shfl_sync(0xffffffffu, pk, src);
      fv = __shfl_sync(0xffffffffu, vk, src);
      return true;
    }
  }
  fg = fp = fv = __longlong_as_double(0x7ff8000000000000LL);
  return false;
}

__global__ void __launch_bounds__(kBlock) fues_kernel(const double* __restrict__ grid, const double* __restrict__ policy,
                                                      const double* __restrict__ value,
                                                      const double* __restrict__ savings, int n_rows, int n_in,
                                                      double thr, int window, double* __restrict__ grid_out,
                                                      double* __restrict__ policy_out, double* __restrict__ value_out,
                                                      int n_out, int* __restrict__ n_kept, double* __restrict__ work) {
  __shared__ int sidx[kMaxSort];
  int np2 = 1;
  while (np2 < n_in) np2 <<= 1;
  const bool use_sav = savings != nullptr;
  for (int row = blockIdx.x; row < n_rows; row += gridDim.x) {
    const double* G = grid + (int64_t)row * n_in;
    const double* P = policy + (int64_t)row * n_in;
    const double* V = value + (int64_t)row * n_in;
    const double* S = use_sav ? savings + (int64_t)row * n_in : nullptr;
    double* g = work + (int64_t)row * 4 * n_in;
    double* p = g + n_in;
    double* v = p + n_in;
    double* s = v + n_in;
    // ---- 1. bitonic sort of indices by the lexsort key
    __syncthreads();
    for (int t = threadIdx.x; t < np2; t += kBlock) sidx[t] = t;
    __syncthreads();
    for (int size = 2; size <= np2; size <<= 1) {
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int t = threadIdx.x; t < np2; t += kBlock) {
          const int partner = t ^ stride;
          if (partner > t) {
            const bool ascending = (t & size) == 0;
            const Key a = load_key(G, V, P, sidx[t], n_in);
            const Key b = load_key(G, V, P, sidx[partner], n_in);
            const bool swap = ascending ? key_less(b, a) : key_less(a, b);
            if (swap) {
              const int tmp = sidx[t];
              sidx[t] = sidx[partner];
              sidx[partner] = tmp;
            }
          }
        }
        __syncthreads();
      }
    }
    for (int t = threadIdx.x; t < n_in; t += kBlock) {
      const int i = sidx[t];
      g[t] = G[i];
      p[t] = P[i];
      v[t] = V[i];
      s[t] = use_sav ? S[i] : G[i] - P[i];
    }
    __syncthreads();
    // ---- 2. coincident groups: keep the maximisers, one per savings source
    for (int t = threadIdx.x; t < n_in; t += kBlock) {
      const double gt = g[t];
      bool keep = !isnan_(gt);
      if (keep) {
        int lo = t, hi = t;
        while (lo > 0 && g[lo - 1] == gt) --lo;
        while (hi + 1 < n_in && g[hi + 1] == gt) ++hi;
        if (hi > lo) {
          double vmax = -__longlong_as_double(0x7ff0000000000000LL);
          for (int k = lo; k <= hi; ++k) {
            const double vk = v[k];
            if (!isnan_(vk) && vk > vmax) vmax = vk;
          }
          keep = v[t] == vmax;
          if (keep) {
            for (int k = lo; k < t; ++k)
              if (v[k] == vmax && s[k] == s[t]) keep = false;
          }
        }
      }
      sidx[t] = keep ? 1 : 0;  // reuse shared memory as the keep mask
    }
    __syncthreads();
    for (int t = threadIdx.x; t < n_in; t += kBlock) {
      if (!sidx[t]) {
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
        g[t] = p[t] = v[t] = s[t] = nan;
      }
    }
    __syncthreads();
    // ---- 3. the scan (warp 0; all lanes hold the state, lane 0 writes)
    if (threadIdx.x < 32) {
      const int lane = threadIdx.x;
      double* GO = grid_out + (int64_t)row * n_out;
      double* PO = policy_out + (int64_t)row * n_out;
      double* VO = value_out + (int64_t)row * n_out;
      const double nan = __longlong_as_double(0x7ff8000000000000LL);
      for (int t = lane; t < n_out; t += 32) GO[t] = PO[t] = VO[t] = nan;
      __syncwarp();
      int cnt = 0;
      auto emit = [&](double eg, double ep, double ev) {
        if (lane == 0 && cnt < n_out) {
          GO[cnt] = eg;
          PO[cnt] = ep;
          VO[cnt] = ev;
        }
        ++cnt;
      };
      double gk = g[0], pk = p[0], vk = v[0];
      double gj = g[0], pj = p[0], vj = v[0], sj = s[0];
      const double near = 16.0 * 2.220446049250313e-16;
      for (int idx = 1; idx < n_in; ++idx) {
        const double gi = g[idx], pi = p[idx], vi = v[idx], si = s[idx];
        const bool valid = !isnan_(gi) && !isnan_(vi);
        const bool sw = valid && policy_jump(gj, pj, gi, pi, thr, true, sj, si);
        const bool node_crossing = valid && sw && gi == gj && vi == vj;
        const double secant = slope(gj, vj, gi, vi);
        const double grad_before = slope(gk, vk, gj, vj);
        double jg, jp, jv;
        const bool jf = find_same_segment(g, p, v, n_in, gj, pj, idx, 1, thr, window, jg, jp, jv);
        bool below_j = false;
        if (sw && jf) below_j = (gi == jg) ? (vi < jv) : (secant < slope(gi, vi, jg, jv));
        const bool sav_dec = si < sj;
        bool dropped = !valid || ((vi < vj) && !sw) || (sav_dec && secant < grad_before) || below_j;
        dropped = dropped && !node_crossing;
        if (dropped) continue;
        double fg, fp, fv, bg, bp, bv;
        const bool ff = find_same_segment(g, p, v, n_in, gi, pi, idx, 1, thr, window, fg, fp, fv);
        const bool bf = find_same_segment(g, p, v, n_in, gi, pi, idx, -1, thr, window, bg, bp, bv);
        const bool found = ff || bf;
        const double pg = ff ? fg : bg, pp = ff ? fp : bp, pv = ff ? fv : bv;
        const double i_slope = slope(gi, vi, pg, pv);
        const double i_pslope = slope(gi, pi, pg, pp);
        const bool j_dom = sw && found && (secant > i_slope) && !node_crossing;
        const double pslope_kj = slope(gk, pk, gj, pj);
        double k6g, k6v;
        intersect(gj, vj, grad_before, gi, vi, i_slope, k6g, k6v);
        const double k6pl = pj + pslope_kj * (k6g - gj);
        const double k6pr = pi + i_pslope * (k6g - gi);
        const bool kink6 = j_dom && (k6g > gk) && (k6g < gj) && (k6g < gi);
        const double j_slope = jf ? slope(gj, vj, jg, jv) : grad_before;
        const double j_pslope = jf ? slope(gj, pj, jg, jp) : pslope_kj;
        double k5g, k5v;
        intersect(gj, vj, j_slope, gi, vi, i_slope, k5g, k5v);
        const double k5pl = pj + j_pslope * (k5g - gj);
        const double k5pr = pi + i_pslope * (k5g - gi);
        const bool crossing = !j_dom && !node_crossing && sw && found;
        const double tol = near * fmax(fmax(fabs(gj), fabs(gi)), 1.0);
        const bool on_j = crossing && fabs(k5g - gj) <= tol;
        const bool on_i = crossing && !on_j && fabs(k5g - gi) <= tol;
        const bool kink5 = crossing && !on_j && !on_i && (k5g > gj) && (k5g < gi);
        const bool plain = !j_dom && !kink5 && !on_j && !on_i;
        if (kink6) {
          emit(k6g, k6pl, k6v);
          emit(k6g, k6pr, k6v);
        } else if (plain || kink5 || on_j || on_i) {
          emit(gj, pj, vj);
          if (kink5) {
            emit(k5g, k5pl, k5v);
            emit(k5g, k5pr, k5v);
          } else if (on_j) {
            emit(gj, k5pr, k5v);
          } else if (on_i) {
            emit(gi, k5pl, k5v);
          }
        }
        const bool keeps_k = j_dom && !kink6;
        if (!keeps_k) {
          if (kink5) {
            gk = k5g; pk = k5pr; vk = k5v;
          } else if (kink6) {
            gk = k6g; pk = k6pr; vk = k6v;
          } else {
            gk = gj;
            pk = on_j ? k5pr : pj;
            vk = on_j ? k5v : vj;
          }
        }
        gj = gi; pj = pi; vj = vi; sj = si;
      }
      if (!isnan_(gj) && !isnan_(vj)) emit(gj, pj, vj);
      if (lane == 0) n_kept[row] = cnt;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Shared-memory form (rows of up to kSmemMaxN candidates).
//
// Same three stages and the same decisions as fues_kernel, with the row in
// shared memory and the serial part cut to what it needs:
//   * DC-EGM candidates arrive almost sorted (a value kink sends the
//     endogenous grid back once; on the 2000-point retirement model 0 to 23
//     descents in a row of 2020): an ascending row is not sorted at all, one
//     of up to kMaxRuns ascending runs is merged by ranks (each candidate
//     counts the smaller ones of every other run by binary search), and only
//     a row of more runs goes through the bitonic network;
//   * a step without a policy jump between j and i never reads the
//     look-ahead, the intersections or i's own neighbours -- it is dropped or
//     emits j and shifts (k, j) <- (j, i).  Whether that step is plain (keeps
//     its candidate and only emits j) while j and k are the two candidates
//     before it depends on the position alone: all threads put that bit in a
//     mask, and the scan (warp 0) commits the run up to the next clear bit at
//     once;
//   * the policy-jump test divides only where a product with a rounding
//     margin cannot decide it (policy_jump_fast);
//   * the look-ahead searches run only on steps with a policy jump, 32
//     candidates first, then 128 per step, and j's is kept while j stays;
//   * candidates dropped one after the other are dropped 32 at a time;
//   * the refined rows' NaN tail is filled after the scan, once.
// Every decision is the one fues_kernel takes and every emitted value is
// computed with the same operations and operands, so the rows are identical.
//
// What bounds it: the serial scan of the rows with many policy jumps (a few
// rows of a launch; about 1.5 thousand cycles per jump, in dependent loads,
// ballots and divisions) and the staging.  The row takes as little shared
// memory as it can -- four doubles and an index per candidate, the sort keys
// in the savings' place -- for three CTAs per SM at rows of 2020.  B200, 1056
// rows of 2020 candidates per period (20 periods of the retirement model,
// batch 32): 13.9 ms with a bitonic sort of every row and a step-by-step scan,
// 7.4 ms in this form; with taste shocks (777 points, batch 12, 10 periods)
// 1.76 and 0.57 ms.  Two CTAs per SM with 128 registers: 7.4 ms.  Searching
// the neighbours of every jump ahead of the scan by all warps: slower (10 ms),
// most of them are dropped without it.
constexpr int kSmemMaxN = 4096;
constexpr int kFuesItemWords = 13;

__host__ __device__ constexpr size_t fues_smem_bytes(int n) {
  int np2 = 1;
  while (np2 < n) np2 <<= 1;
  return (size_t)3 * n * sizeof(double) + (size_t)np2 * (sizeof(unsigned long long) + sizeof(unsigned short));
}

// Monotone 64-bit image of a grid value for the sort: NaN ranks with +inf and
// -0 with +0, as the (double) comparison of the lexsort key treats them.
__device__ __forceinline__ unsigned long long grid_key(double g) {
  if (isnan_(g)) g = __longlong_as_double(0x7ff0000000000000LL);
  if (g == 0.0) g = 0.0;
  const unsigned long long b = (unsigned long long)__double_as_longlong(g);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ULL);
}

struct FuesRowIO {
  const double* G;
  const double* P;
  const double* V;
  const double* S;
  double* GO;
  double* PO;
  double* VO;
  int* nk;
  int n_in;
  int n_out;
  double thr;
  int window;  // look-ahead positions inspected in each direction
};

struct FuesContig {
  const double* grid;
  const double* policy;
  const double* value;
  const double* savings;
  double* go;
  double* po;
  double* vo;
  int* nk;
  int n_rows, n_in, n_out;
  double thr;
  int window;
  __device__ __forceinline__ int count() const { return n_rows; }
  __device__ __forceinline__ FuesRowIO row(int r) const {
    FuesRowIO io;
    io.G = grid + (int64_t)r * n_in;
    io.P = policy + (int64_t)r * n_in;
    io.V = value + (int64_t)r * n_in;
    io.S = savings ? savings + (int64_t)r * n_in : nullptr;
    io.GO = go + (int64_t)r * n_out;
    io.PO = po + (int64_t)r * n_out;
    io.VO = vo + (int64_t)r * n_out;
    io.nk = nk + r;
    io.n_in = n_in;
    io.n_out = n_out;
    io.thr = thr;
    io.window = window;
    return io;
  }
};

// item words: 0 grid, 1 policy, 2 value, 3 savings (0: none), 4 grid_out,
// 5 policy_out, 6 value_out, 7 n_kept (int32), 8 n_rows, 9 n_in, 10 n_out,
// 11 jump_thresh (double bits), 12 look-ahead window (<= 0: exhaustive);
// one tile per row
struct FuesItems {
  const int64_t* items;
  const int* prefix;
  int n_items, n_tiles;
  __device__ __forceinline__ int count() const { return n_tiles; }
  __device__ __forceinline__ FuesRowIO row(int tile) const {
    int lo = 0, hi = n_items - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (prefix[mid] <= tile) lo = mid; else hi = mid - 1;
    }
    const int64_t* it = items + (int64_t)lo * kFuesItemWords;
    const int r = tile - prefix[lo];
    FuesRowIO io;
    io.n_in = (int)it[9];
    io.n_out = (int)it[10];
    io.thr = __longlong_as_double(it[11]);
    io.window = it[12] > 0 ? (int)it[12] : io.n_in;
    io.G = reinterpret_cast<const double*>(it[0]) + (int64_t)r * io.n_in;
    io.P = reinterpret_cast<const double*>(it[1]) + (int64_t)r * io.n_in;
    io.V = reinterpret_cast<const double*>(it[2]) + (int64_t)r * io.n_in;
    io.S = it[3] ? reinterpret_cast<const double*>(it[3]) + (int64_t)r * io.n_in : nullptr;
    io.GO = reinterpret_cast<double*>(it[4]) + (int64_t)r * io.n_out;
    io.PO = reinterpret_cast<double*>(it[5]) + (int64_t)r * io.n_out;
    io.VO = reinterpret_cast<double*>(it[6]) + (int64_t)r * io.n_out;
    io.nk = reinterpret_cast<int*>(it[7]) + r;
    return io;
  }
};

constexpr int kPerThread = kSmemMaxN / kBlock;  // candidates a thread holds in registers
constexpr int kMaxRuns = 17;                    // ascending runs merged by ranks
constexpr int kMaxSegments = 64;                // runs of plain steps copied by the whole CTA

// x[t] <- x[sidx[t]] for t < n, through registers
__device__ __forceinline__ void permute_sorted(double* x, const unsigned short* sidx, int n) {
  double r[kPerThread];
#pragma unroll
  for (int k = 0; k < kPerThread; ++k) {
    const int t = threadIdx.x + k * kBlock;
    if (t < n) r[k] = x[sidx[t]];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kPerThread; ++k) {
    const int t = threadIdx.x + k * kBlock;
    if (t < n) x[t] = r[k];
  }
}

// policy_jump with the division only near the threshold: with t = thr |dx|
// rounded once, |dy| beyond t (1 +- 1e-15) decides |dy / dx| > thr, however
// the quotient rounds.
__device__ __forceinline__ bool policy_jump_fast(double ga, double pa, double gb, double pb, double thr,
                                                 bool use_sav, double sa, double sb) {
  const double ia = ga - pa, ib = gb - pb;
  if (ga == gb) return use_sav ? (sa != sb) : (ia != ib);
  const double ad = fabs(ib - ia), t = thr * fabs(gb - ga);
  if (t > 1e-290 && t < 1e300) {
    if (ad > t * (1.0 + 1e-15)) return true;
    if (ad < t * (1.0 - 1e-15)) return false;
  }
  return fabs(slope(ga, ia, gb, ib)) > thr;
}

// find_same_segment over shared memory: position of the nearest same-segment
// candidate of (ag, ap) from idx in direction dir within `window` positions,
// -1 if there is none (warp-cooperative; 32 candidates, then 128 at a time)
__device__ __forceinline__ int find_same_segment_at(const double* g, const double* p, const double* v, int n,
                                                    double ag, double ap, int idx, int dir, double thr, int window) {
  const int lane = threadIdx.x & 31;
  const int last = min(window, dir > 0 ? n - 1 - idx : idx);  // offsets 1 .. last
  auto same = [&](int off) {
    bool ok = false;
    if (off <= last) {
      const int k = idx + dir * off;
      const double gk = g[k];
      ok = !isnan_(gk) && !isnan_(v[k]) && !policy_jump_fast(ag, ap, gk, p[k], thr, false, 0.0, 0.0);
    }
    return ok;
  };
  if (last < 1) return -1;
  unsigned m = __ballot_sync(0xffffffffu, same(1 + lane));
  if (m) return idx + dir * __ffs(m);
  for (int base = 33; base <= last; base += 128) {
    unsigned b[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) b[q] = __ballot_sync(0xffffffffu, same(base + 32 * q + lane));
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (b[q]) return idx + dir * (base + 32 * q + __ffs(b[q]) - 1);
  }
  return -1;
}

template <class Rows>
__global__ void __launch_bounds__(kBlock, 3) fues_smem_kernel(Rows rows) {
  extern __shared__ __align__(16) unsigned char fues_smem[];
  __shared__ unsigned plain_mask[kSmemMaxN / 32 + 1];
  __shared__ int run_start[kMaxRuns];
  __shared__ int3 segs[kMaxSegments];  // runs of plain steps to copy
  __shared__ int n_desc, n_emit, n_runs;
  const int total = rows.count();
  const double nan = __longlong_as_double(0x7ff8000000000000LL);
  const int tid = threadIdx.x, lane = tid & 31;
  for (int row = blockIdx.x; row < total; row += gridDim.x) {
    const FuesRowIO io = rows.row(row);
    const int n = io.n_in;
    const int n_out = io.n_out;
    const double thr = io.thr;
    const double* __restrict__ G = io.G;
    const double* __restrict__ P = io.P;
    const double* __restrict__ V = io.V;
    const double* __restrict__ S = io.S;
    int np2 = 1;
    while (np2 < n) np2 <<= 1;
    // three arrays of n, then np2 words for the savings (the bitonic network's
    // keys while it sorts), then the order
    double* g = reinterpret_cast<double*>(fues_smem);
    double* p = g + n;
    double* v = p + n;
    double* s = v + n;
    unsigned long long* skey = reinterpret_cast<unsigned long long*>(s);
    unsigned short* sidx = reinterpret_cast<unsigned short*>(skey + np2);
    __syncthreads();  // the previous row is done with shared memory
    // ---- 1. stage the row (input order), four candidates per thread in flight
    if (tid == 0) n_desc = 0;
    for (int t0 = tid; t0 < n; t0 += 4 * kBlock) {
      double a[4], b[4], c[4], d[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int t = t0 + q * kBlock;
        if (t < n) {
          a[q] = __ldg(G + t);
          b[q] = __ldg(P + t);
          c[q] = __ldg(V + t);
          d[q] = S ? __ldg(S + t) : 0.0;
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int t = t0 + q * kBlock;
        if (t < n) {
          g[t] = a[q];
          p[t] = b[q];
          v[t] = c[q];
          s[t] = S ? d[q] : a[q] - b[q];
        }
      }
    }
    __syncthreads();
    // does position a's candidate come before position b's?
    auto before = [&](int a, int b) { return !key_less(load_key(g, v, p, b, n), load_key(g, v, p, a, n)); };
    for (int t = tid; t + 1 < n; t += kBlock) {
      if (!before(t, t + 1)) {
        const int q = atomicAdd(&n_desc, 1);
        if (q < kMaxRuns - 1) run_start[q] = t + 1;
      }
    }
    __syncthreads();
    const int nd = n_desc;
    if (nd > 0) {
      for (int t = tid; t < np2; t += kBlock) skey[t] = t < n ? grid_key(g[t]) : ~0ULL;  // padding sorts last
      __syncthreads();
    }
    if (nd > 0 && nd < kMaxRuns) {
      // ranks: own place in the run plus, per other run, the candidates
      // before this one
      if (tid == 0) {
        for (int a = 1; a < nd; ++a) {
          const int x = run_start[a];
          int b = a;
          for (; b > 0 && run_start[b - 1] > x; --b) run_start[b] = run_start[b - 1];
          run_start[b] = x;
        }
      }
      __syncthreads();
      for (int t = tid; t < n; t += kBlock) {
        const unsigned long long key = skey[t];
        int rank = 0, r0 = 0;
        for (int r = 0; r <= nd; ++r) {
          const int r1 = r < nd ? run_start[r] : n;
          if (t >= r0 && t < r1) {
            rank += t - r0;
          } else {
            int lo = r0, hi = r1;  // first of the run that does not come before t
            while (lo < hi) {
              const int mid = (lo + hi) >> 1;
              const unsigned long long km = skey[mid];
              if (km != key ? km < key : before(mid, t)) lo = mid + 1; else hi = mid;
            }
            rank += lo - r0;
          }
          r0 = r1;
        }
        sidx[rank] = (unsigned short)t;
      }
      __syncthreads();
    } else if (nd >= kMaxRuns) {
      // bitonic network over (key, index) pairs: a compare-exchange reads
      // positions t and t ^ stride; only equal grid keys consult value,
      // policy and index
      for (int t = tid; t < np2; t += kBlock) {
        sidx[t] = (unsigned short)t;
      }
      __syncthreads();
      const int half = np2 >> 1;
      for (int size = 2; size <= np2; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
          const int ls = __ffs(stride) - 1;  // stride = 2^ls
#pragma unroll 4
          for (int j = tid; j < half; j += kBlock) {
            // the j-th compare-exchange pair (t, t + stride) of this stage:
            // the positions whose bit ls is clear, in order
            const int t = ((j >> ls) << (ls + 1)) | (j & (stride - 1));
            const int partner = t + stride;
            const bool ascending = (t & size) == 0;
            const unsigned long long ka = skey[t], kb = skey[partner];
            const unsigned short ia = sidx[t], ib = sidx[partner];
            bool a_first;  // does (ka, ia) come before (kb, ib)?
            if (ka != kb) {
              a_first = ka < kb;
            } else {
              a_first = !key_less(load_key(g, v, p, ib, n), load_key(g, v, p, ia, n));
            }
            if (ascending != a_first) {
              skey[t] = kb;
              skey[partner] = ka;
              sidx[t] = ib;
              sidx[partner] = ia;
            }
          }
          __syncthreads();
        }
      }
    }
    if (nd > 0) {
      permute_sorted(g, sidx, n);
      permute_sorted(p, sidx, n);
      permute_sorted(v, sidx, n);
      __syncthreads();  // the savings come back in place of the keys
      for (int t = tid; t < n; t += kBlock) s[t] = S ? __ldg(S + sidx[t]) : g[t] - p[t];
      __syncthreads();
    }
    // ---- 2. coincident groups: keep the maximisers, one per savings source
    unsigned drop_bits = 0u;  // bit k: the thread's k-th position goes
    for (int k = 0, t = tid; t < n; ++k, t += kBlock) {
      const double gt = g[t];
      bool keep = !isnan_(gt);
      if (keep) {
        int lo = t, hi = t;
        while (lo > 0 && g[lo - 1] == gt) --lo;
        while (hi + 1 < n && g[hi + 1] == gt) ++hi;
        if (hi > lo) {
          double vmax = -__longlong_as_double(0x7ff0000000000000LL);
          for (int q = lo; q <= hi; ++q) {
            const double vq = v[q];
            if (!isnan_(vq) && vq > vmax) vmax = vq;
          }
          keep = v[t] == vmax;
          if (keep) {
            for (int q = lo; q < t; ++q)
              if (v[q] == vmax && s[q] == s[t]) keep = false;
          }
        }
      }
      if (!keep) drop_bits |= 1u << k;
    }
    __syncthreads();
    for (int k = 0, t = tid; t < n; ++k, t += kBlock) {
      if ((drop_bits >> k) & 1u) g[t] = p[t] = v[t] = s[t] = nan;
    }
    __syncthreads();
    // ---- 3a. plain steps: while j and k are the two candidates before t, the
    // step at t keeps candidate t and only emits j when t is valid, shows no
    // policy jump from t - 1, and is neither below t - 1 nor a savings
    // decrease with a secant under the previous one
    for (int t = tid; t < ((n + 31) & ~31); t += kBlock) {
      bool ok = false;
      if (t >= 2 && t < n) {
        const double gt = g[t], vt = v[t], g1 = g[t - 1], v1 = v[t - 1];
        ok = !isnan_(gt) && !isnan_(vt) && !(vt < v1) &&
             !policy_jump_fast(g1, p[t - 1], gt, p[t], thr, true, s[t - 1], s[t]);
        if (ok && s[t] < s[t - 1]) ok = !(slope(g1, v1, gt, vt) < slope(g[t - 2], v[t - 2], g1, v1));
      }
      const unsigned m = __ballot_sync(0xffffffffu, ok);
      if (lane == 0) plain_mask[t >> 5] = m;
    }
    __syncthreads();
    // ---- 3b. the scan (warp 0; all lanes hold the state, lane 0 writes)
    if (tid < 32) {
      double* GO = io.GO;
      double* PO = io.PO;
      double* VO = io.VO;
      const int words = (n + 31) >> 5;
      int cnt = 0, n_seg = 0;
      auto emit = [&](double eg, double ep, double ev) {
        if (lane == 0 && cnt < n_out) {
          GO[cnt] = eg;
          PO[cnt] = ep;
          VO[cnt] = ev;
        }
        ++cnt;
      };
      double gk = g[0], pk = p[0], vk = v[0];
      double gj = g[0], pj = p[0], vj = v[0], sj = s[0];
      int jidx = 0, kidx = 0;  // candidates j and k are (kidx < 0: k is a kink point)
      const double near = 16.0 * 2.220446049250313e-16;
      const int window = min(io.window, n);
      int jn = -1;    // j's next same-segment candidate, while have_jn
      int seen = -1;  // the last position looked at for it
      bool have_jn = false;
      for (int idx = 1; idx < n; ++idx) {
        // the run of plain steps from idx ends at the next clear bit.  Its
        // first step may follow any k if its savings do not decrease (the
        // only test that reads k); the later ones follow t - 2 and t - 1
        if (jidx == idx - 1 && ((kidx >= 0 && kidx == jidx - 1) || !(s[idx] < sj))) {
          int stop = n;
          for (int w0 = idx >> 5; w0 < words; w0 += 32) {
            unsigned clear = 0u;
            if (w0 + lane < words) {
              clear = ~plain_mask[w0 + lane];
              if (w0 + lane == idx >> 5) clear &= 0xffffffffu << (idx & 31);
            }
            const unsigned b = __ballot_sync(0xffffffffu, clear != 0u);
            if (b) {
              const int src = __ffs(b) - 1;
              const unsigned c = __shfl_sync(0xffffffffu, clear, src);
              stop = min(n, 32 * (w0 + src) + __ffs(c) - 1);
              break;
            }
          }
          const int m = stop - idx;
          if (m > 0) {
            // its j's are copied by the whole CTA after the scan
            if (n_seg < kMaxSegments) {
              if (lane == 0) segs[n_seg] = make_int3(idx - 1, cnt, m);
              ++n_seg;
            } else {
              for (int q = lane; q < m; q += 32) {
                if (cnt + q < n_out) {
                  GO[cnt + q] = g[idx - 1 + q];
                  PO[cnt + q] = p[idx - 1 + q];
                  VO[cnt + q] = v[idx - 1 + q];
                }
              }
            }
            cnt += m;
            const int nj = idx + m - 1;
            gk = g[nj - 1]; pk = p[nj - 1]; vk = v[nj - 1];
            kidx = nj - 1;
            gj = g[nj]; pj = p[nj]; vj = v[nj]; sj = s[nj];
            jidx = nj;
            have_jn = false;
            idx = nj;  // the loop's increment moves to the first step not in the run
            continue;
          }
        }
        // A dropped candidate leaves j and k as they are, so the lanes test
        // idx .. idx + 31 against them at once and the warp drops the leading
        // run.  j's next same-segment candidate jn is the same for every t
        // before it; a bounded look-ahead sees it from t within its window
        // (one candidate at a time, 200 rows of 2020 with 12 kinks took 1063 us
        // at a window of 10, 32 at a time 564).
        const int t = idx + lane;
        const bool in = t < n;
        const double gt = in ? g[t] : nan, vt = in ? v[t] : nan, pt = in ? p[t] : nan, st = in ? s[t] : nan;
        const bool valid = !isnan_(gt) && !isnan_(vt);
        const bool jump = valid && policy_jump_fast(gj, pj, gt, pt, thr, true, sj, st);
        const unsigned jumps = __ballot_sync(0xffffffffu, jump);
        if (jumps && !(have_jn && (jn > idx || (jn < 0 && seen >= min(n - 1, idx + 31 + window))))) {
          const bool same = valid && lane > 0 && (gt == gj ? (gj - pj == gt - pt) : !jump);
          const unsigned ms = __ballot_sync(0xffffffffu, same);
          jn = ms ? idx + __ffs(ms) - 1 : find_same_segment_at(g, p, v, n, gj, pj, idx + 31, 1, thr, window);
          seen = idx + 31 + window;
          have_jn = true;
        }
        const bool ahead = jumps != 0u && jn >= 0;
        const double jg = ahead ? g[jn] : nan, jp = ahead ? p[jn] : nan, jv = ahead ? v[jn] : nan;
        const bool sees = ahead && jn - t <= window;
        bool drop = (vt < vj) && !jump;
        if (valid && !drop && (st < sj || (jump && sees))) {
          const double sec_t = slope(gj, vj, gt, vt);
          if (st < sj) drop = sec_t < slope(gk, vk, gj, vj);
          if (!drop && jump && sees) drop = (gt == jg) ? (vt < jv) : (sec_t < slope(gt, vt, jg, jv));
        }
        const bool open = jump && ahead && t >= jn;  // needs the candidate after jn
        const bool node = jump && gt == gj && vt == vj;
        const unsigned stays = ~__ballot_sync(0xffffffffu, in && (!valid || (drop && !node && !open)));
        const unsigned keeps = __ballot_sync(0xffffffffu, valid && !jump && !drop);
        const int m = stays ? __ffs(stays) - 1 : 32;
        const bool keep = m < 32 && ((keeps >> m) & 1u);
        if (m > 0 || keep) {
          idx += m;
          if (keep) {  // the first one not dropped shows no jump: it only emits j
            emit(gj, pj, vj);
            gk = gj;
            pk = pj;
            vk = vj;
            kidx = jidx;
            gj = g[idx];
            pj = p[idx];
            vj = v[idx];
            sj = s[idx];
            jidx = idx;
            have_jn = false;
          } else {
            --idx;
          }
          continue;
        }
        // a kept candidate across a policy jump
        const bool jf = ahead && jn - idx <= window;
        const double gi = g[idx], vi = v[idx], pi = p[idx], si = s[idx];
        const bool node_crossing = gi == gj && vi == vj;
        have_jn = false;  // j changes
        const double sc = slope(gj, vj, gi, vi);
        const double gb = slope(gk, vk, gj, vj);
        // i's own neighbour: forward, or backward where there is none
        int nb = find_same_segment_at(g, p, v, n, gi, pi, idx, 1, thr, io.window);
        if (nb < 0) nb = find_same_segment_at(g, p, v, n, gi, pi, idx, -1, thr, io.window);
        const bool found = nb >= 0;
        const double pg = found ? g[nb] : nan, pp = found ? p[nb] : nan, pv = found ? v[nb] : nan;
        const double i_slope = slope(gi, vi, pg, pv);
        const double i_pslope = slope(gi, pi, pg, pp);
        const bool j_dom = found && (sc > i_slope) && !node_crossing;
        const double pslope_kj = slope(gk, pk, gj, pj);
        double k6g, k6v;
        intersect(gj, vj, gb, gi, vi, i_slope, k6g, k6v);
        const double k6pl = pj + pslope_kj * (k6g - gj);
        const double k6pr = pi + i_pslope * (k6g - gi);
        const bool kink6 = j_dom && (k6g > gk) && (k6g < gj) && (k6g < gi);
        const double j_slope = jf ? slope(gj, vj, jg, jv) : gb;
        const double j_pslope = jf ? slope(gj, pj, jg, jp) : pslope_kj;
        double k5g, k5v;
        intersect(gj, vj, j_slope, gi, vi, i_slope, k5g, k5v);
        const double k5pl = pj + j_pslope * (k5g - gj);
        const double k5pr = pi + i_pslope * (k5g - gi);
        const bool crossing = !j_dom && !node_crossing && found;
        const double tol = near * fmax(fmax(fabs(gj), fabs(gi)), 1.0);
        const bool on_j = crossing && fabs(k5g - gj) <= tol;
        const bool on_i = crossing && !on_j && fabs(k5g - gi) <= tol;
        const bool kink5 = crossing && !on_j && !on_i && (k5g > gj) && (k5g < gi);
        const bool plain = !j_dom && !kink5 && !on_j && !on_i;
        if (kink6) {
          emit(k6g, k6pl, k6v);
          emit(k6g, k6pr, k6v);
        } else if (plain || kink5 || on_j || on_i) {
          emit(gj, pj, vj);
          if (kink5) {
            emit(k5g, k5pl, k5v);
            emit(k5g, k5pr, k5v);
          } else if (on_j) {
            emit(gj, k5pr, k5v);
          } else if (on_i) {
            emit(gi, k5pl, k5v);
          }
        }
        const bool keeps_k = j_dom && !kink6;
        if (!keeps_k) {
          if (kink5) {
            gk = k5g; pk = k5pr; vk = k5v; kidx = -1;
          } else if (kink6) {
            gk = k6g; pk = k6pr; vk = k6v; kidx = -1;
          } else {
            gk = gj;
            pk = on_j ? k5pr : pj;
            vk = on_j ? k5v : vj;
            kidx = on_j ? -1 : jidx;
          }
        }
        gj = gi; pj = pi; vj = vi; sj = si;
        jidx = idx;
      }
      if (!isnan_(gj) && !isnan_(vj)) emit(gj, pj, vj);
      if (lane == 0) {
        *io.nk = cnt;
        n_emit = cnt;
        n_runs = n_seg;
      }
    }
    __syncthreads();
    for (int r = 0; r < n_runs; ++r) {
      const int3 seg = segs[r];  // (first position, first output, points)
      const int m = min(seg.z, n_out - seg.y);
      for (int q = tid; q < m; q += kBlock) {
        io.GO[seg.y + q] = g[seg.x + q];
        io.PO[seg.y + q] = p[seg.x + q];
        io.VO[seg.y + q] = v[seg.x + q];
      }
    }
    for (int t = n_emit + tid; t < n_out; t += kBlock) io.GO[t] = io.PO[t] = io.VO[t] = nan;
  }
}

// the dynamic shared-memory limit of both instantiations, set once per device
std::mutex g_attr_mu;
bool g_attr_done[64] = {};

int fues_smem_attr(std::string& err) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) {
    err = "fues: device ordinal >= 64";
    return LCMX_ERR_ARGS;
  }
  std::lock_guard<std::mutex> g(g_attr_mu);
  if (g_attr_done[dev]) return LCMX_OK;
  const int bytes = (int)fues_smem_bytes(kSmemMaxN);
  cudaError_t e = cudaFuncSetAttribute(fues_smem_kernel<FuesContig>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(fues_smem_kernel<FuesItems>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) {
    err = std::string("fues: shared-memory attribute: ") + cudaGetErrorString(e);
    return LCMX_ERR_CUDA;
  }
  g_attr_done[dev] = true;
  return LCMX_OK;
}

int fues_grid(int rows) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return rows < sms * 16 ? rows : sms * 16;
}

}  // namespace

extern "C" size_t lcmx_fues_workspace_bytes(int n_rows, int n_in) {
  if (n_rows <= 0 || n_in <= 0) return 0;
  return (size_t)n_rows * 4 * (size_t)n_in * sizeof(double);
}

static int launch_fues(const double* grid, const double* policy, const double* value, const double* savings,
                       int n_rows, int n_in, double jump_thresh, int window, double* grid_out,
                       double* policy_out, double* value_out, int n_out, int* n_kept, double* work,
                       cudaStream_t stream, std::string& err) {
  if (window <= 0) window = n_in;  // exhaustive look-ahead
  if (n_in <= kSmemMaxN) {
    int rc = fues_smem_attr(err);
    if (rc) return rc;
    FuesContig rows{grid, policy, value, savings, grid_out, policy_out, value_out, n_kept,
                    n_rows, n_in, n_out, jump_thresh, window};
    fues_smem_kernel<FuesContig><<<fues_grid(n_rows), kBlock, fues_smem_bytes(n_in), stream>>>(rows);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      err = std::string("fues launch: ") + cudaGetErrorString(e);
      return LCMX_ERR_LAUNCH;
    }
    return LCMX_OK;
  }
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int grid_n = n_rows < sms * 4 ? n_rows : sms * 4;
  fues_kernel<<<grid_n, kBlock, 0, stream>>>(grid, policy, value, savings, n_rows, n_in, jump_thresh, window,
                                             grid_out, policy_out, value_out, n_out, n_kept, work);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    err = std::string("fues launch: ") + cudaGetErrorString(e);
    return LCMX_ERR_LAUNCH;
  }
  return LCMX_OK;
}

int lcmx_set_error_from(lcmx_ctx* ctx, int code, const std::string& msg);

extern "C" int lcmx_fues_scan(lcmx_ctx* ctx, const double* grid, const double* policy, const double* value,
                              const double* savings, int n_rows, int n_in, double jump_thresh,
                              int n_points_to_scan, double* grid_out, double* policy_out, double* value_out,
                              int n_out, int* n_kept, void* workspace, size_t workspace_bytes, void* stream) {
  if (!ctx || !grid || !policy || !value || !grid_out || !policy_out || !value_out || !n_kept || n_rows < 0 ||
      n_in < 1 || n_out < 1 || !(jump_thresh > 0.0))
    return lcmx_set_error_from(ctx, LCMX_ERR_ARGS, "lcmx_fues_scan: bad arguments");
  if (n_in > kMaxSort)
    return lcmx_set_error_from(ctx, LCMX_ERR_ARGS, "lcmx_fues_scan: rows longer than 8192 candidates");
  if (n_rows == 0) return LCMX_OK;
  if (!workspace || workspace_bytes < lcmx_fues_workspace_bytes(n_rows, n_in))
    return lcmx_set_error_from(ctx, LCMX_ERR_ARGS, "lcmx_fues_scan: workspace too small");
  std::string err;
  int rc = launch_fues(grid, policy, value, savings, n_rows, n_in, jump_thresh, n_points_to_scan, grid_out,
                       policy_out, value_out, n_out, n_kept, static_cast<double*>(workspace), (cudaStream_t)stream,
                       err);
  if (rc) return lcmx_set_error_from(ctx, rc, err);
  return LCMX_OK;
}

// ---------------------------------------------------------------------------
// Variant that allocates nothing.
//
// Some callers cannot call cudaMalloc on this path: code running inside
// another runtime's execution -- for example an XLA FFI custom-call handler,
// which is how the reference runs its native kernels -- must not allocate
// there (cudaMalloc synchronises the device and bypasses the runtime's
// allocator).  For them lcmx_fues_scan_static takes its workspace from the
// file-scope device array below instead of a caller pointer.
//
// * Size: kStaticScratchBytes (8 MiB) per device, held by every GPU that
//   loads this library until the process exits.  A call needs
//   lcmx_fues_workspace_bytes(n_rows, n_in) <= 8 MiB, i.e. at most
//   262144 / n_in rows (129 rows of 2020 candidates); larger calls are
//   rejected with LCMX_ERR_ARGS.
// * Set-up: the first call on a device, with that device current, looks up
//   the array's device address with cudaGetSymbolAddress (in host code the
//   symbol is only a host-side stand-in, not a device address) and caches it
//   for that device.  Make that first call before any stream capture.  Each
//   call makes the context's device current for the lookup and the launch and
//   then restores the caller's current device.
// * Which rows touch the array: rows of up to 4096 candidates are staged in
//   shared memory and leave it unused; rows of 4097..8192 candidates go
//   through the global-workspace kernel, whose per-row sorted copy lives in
//   the array.
// * Sharing: every call uses the same array, which keeps the last call's
//   contents.  Nothing in it has to start at zero (each row's sorted copy is
//   written in full before it is read), but calls that overlap on the GPU
//   race on it: serialise them (one stream, or events).
namespace {
constexpr size_t kStaticScratchBytes = size_t(8) << 20;
__device__ __align__(256) double g_fues_static_scratch[kStaticScratchBytes / sizeof(double)];
std::mutex g_static_mu;
double* g_static_ptr[64] = {};
}  // namespace

int lcmx_ctx_device_of(const lcmx_ctx* ctx);

extern "C" int lcmx_fues_scan_static(lcmx_ctx* ctx, const double* grid, const double* policy, const double* value,
                                     const double* savings, int n_rows, int n_in, double jump_thresh,
                                     double* grid_out, double* policy_out, double* value_out, int n_out,
                                     int* n_kept, void* stream) {
  if (!ctx || !grid || !policy || !value || !grid_out || !policy_out || !value_out || !n_kept || n_rows < 0 ||
      n_in < 1 || n_out < 1 || !(jump_thresh > 0.0))
    return lcmx_set_error_from(ctx, LCMX_ERR_ARGS, "lcmx_fues_scan_static: bad arguments");
  if (n_in > kMaxSort)
    return lcmx_set_error_from(ctx, LCMX_ERR_ARGS, "lcmx_fues_scan_static: rows longer than 8192 candidates");
  const size_t need = lcmx_fues_workspace_bytes(n_rows, n_in);
  if (need > kStaticScratchBytes)
    return lcmx_set_error_from(
        ctx, LCMX_ERR_ARGS,
        "lcmx_fues_scan_static: " + std::to_string(n_rows) + " rows of " + std::to_string(n_in) +
            " candidates need " + std::to_string(need) + " bytes of scratch, more than the 8 MiB static array (at most " +
            std::to_string(kStaticScratchBytes / (4 * sizeof(double) * (size_t)n_in)) + " rows of this length)");
  if (n_rows == 0) return LCMX_OK;
  const int dev = lcmx_ctx_device_of(ctx);
  if (dev < 0 || dev >= 64) return lcmx_set_error_from(ctx, LCMX_ERR_ARGS, "lcmx_fues_scan_static: device ordinal >= 64");
  // The context's device is made current for the symbol lookup and the
  // launch; the caller's current device is put back before every return.
  int prev = -1;
  cudaError_t e = cudaGetDevice(&prev);
  if (e != cudaSuccess) return lcmx_set_error_from(ctx, LCMX_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
  if (prev != dev) {
    e = cudaSetDevice(dev);
    if (e != cudaSuccess) return lcmx_set_error_from(ctx, LCMX_ERR_CUDA, std::string("cudaSetDevice: ") + cudaGetErrorString(e));
  }
  int rc = LCMX_OK;
  std::string err;
  double* work = nullptr;
  {
    std::lock_guard<std::mutex> g(g_static_mu);
    if (!g_static_ptr[dev]) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_fues_static_scratch);
      if (e != cudaSuccess || !p) {
        rc = LCMX_ERR_CUDA;
        err = std::string("cudaGetSymbolAddress(static FUES scratch): ") + cudaGetErrorString(e);
      } else {
        g_static_ptr[dev] = static_cast<double*>(p);
      }
    }
    work = g_static_ptr[dev];
  }
  if (rc == LCMX_OK)
    rc = launch_fues(grid, policy, value, savings, n_rows, n_in, jump_thresh, 0, grid_out, policy_out, value_out,
                     n_out, n_kept, work, (cudaStream_t)stream, err);
  if (prev != dev) cudaSetDevice(prev);
  if (rc) return lcmx_set_error_from(ctx, rc, err);
  return LCMX_OK;
}

// ---------------------------------------------------------------------------
// Item form: the rows of several candidate blocks (one per solve instance)
// in one launch; see FuesItems for the item words.
extern "C" int lcmx_fues_step(lcmx_ctx* ctx, const void* items, const int* tile_prefix, int n_items, int n_rows,
                              int max_n_in, void* stream) {
  if (!ctx || n_items < 0 || n_rows < 0 || (n_items > 0 && (!items || !tile_prefix)))
    return lcmx_set_error_from(ctx, LCMX_ERR_ARGS, "lcmx_fues_step: bad arguments");
  if (max_n_in < 1 || max_n_in > kSmemMaxN)
    return lcmx_set_error_from(ctx, LCMX_ERR_ARGS,
                               "lcmx_fues_step: rows must hold 1.." + std::to_string(kSmemMaxN) + " candidates");
  if (n_items == 0 || n_rows == 0) return LCMX_OK;
  std::string err;
  int rc = fues_smem_attr(err);
  if (rc) return lcmx_set_error_from(ctx, rc, err);
  FuesItems rows{static_cast<const int64_t*>(items), tile_prefix, n_items, n_rows};
  fues_smem_kernel<FuesItems><<<fues_grid(n_rows), kBlock, fues_smem_bytes(max_n_in), (cudaStream_t)stream>>>(rows);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return lcmx_set_error_from(ctx, LCMX_ERR_LAUNCH, std::string("lcmx_fues_step: ") + cudaGetErrorString(e));
  return LCMX_OK;
}
