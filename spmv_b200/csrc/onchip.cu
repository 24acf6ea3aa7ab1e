// CG with the vectors on chip for the batched and the mixed solves (no counterpart
// in the reference; each recurrence is spmv::cg's, cg.cpp:50-80, with the
// FP32-inner / FP64-refinement scheme of the mixed solver).  The mixed solve of one
// matrix is one group over the grid, on the matrix's SELL layout (MX below).
//
// In a batch every unit (a system, or one column of the block of right-hand sides) gets
// its own group of CTAs of one cooperative launch, and the groups iterate
// independently: each has its own counter and partial sums, so nothing waits for
// a larger unit, and a unit that has converged leaves.  A CTA keeps its rows' p
// in shared memory and r, y and d in tensor memory (3 columns per slice in FP32,
// 6 in FP64), each entry with the lane that owns its row, and streams its slices
// through per-warp rings (sell_ring.cuh).  Only p crosses L2: shared memory holds
// it over the window of columns that the CTA's slices gather (the planner's order
// makes that a band around the rows), and the rows of the group's other CTAs are
// copied in, coalesced, before each product; what a window too wide for shared
// memory leaves out is gathered from L2.
//
// Per iteration (the merged update of the fused CG, two syncs of the group):
//   A  y = A p; the sums p.y, r.y, y.y and r.r                     | group sum
//      r.r is that of the true r: the stopping and refinement tests.  If the
//      unit refines, y is not used (R below); else alpha = r.r / p.y and
//      beta = r1.r1 / r.r with r1.r1 = r.r - 2 alpha r.y + alpha^2 y.y
//   C  d += alpha p, r -= alpha y, p = r + beta p                   | group barrier
//   R  x += d, d = 0                                                | group barrier
//      r = fl(b - A64 x) (FP64), q = p - r_old; ||r64||^2, r.r, r.q | group sum
//      p = r + s (q - c r), s = r.r / r_old.r_old, c = r.q / r.r    | group barrier
// which is the lockstep kernel's refinement step: q is the last beta p, s
// corrects that beta for the true residual and c makes the new direction's old
// part orthogonal to it.
//
// What bounds it: 24 mesh systems of 2,048 to 24,000 rows (14 entries per row) and
// a block of 16 columns take 72 us per iteration in the lockstep kernel (grid
// barriers of 296 CTAs, and phases that wait for their slowest CTA) and 11 here
// (22.9 ms a solve against 3.5; FP64 21.0 against 3.7).  24 systems of 22,000 rows:
// 13 us, of which the two syncs and the fixed part of the phases are 6 and the
// rest is 1.2 per slice of the busiest warp (the instructions of the product);
// small systems: 5 us with one CTA, 7 with more.  7 systems of 800 to 3,000 rows
// and 5 columns: 63 us in the lockstep kernel, 5.6 here; 24 of 22,000 and 32
// columns, the chip full, 105 and 24.
// One matrix, mixed (the fused form of ir.cu before): 27-point 96^3 41.3 us per
// iteration, now 28.6 (its entries are 22 at the rate of a copy); 5-point 1024^2
// 17.3 and 14.7, 200 x 180 19.1 and 5.8 (as a CUDA graph before); 27-point 40^3
// 10.7 and 8.1.
#include <algorithm>
#include <cmath>
#include <queue>

#include "batch.h"
#include "sell_ring.cuh"

namespace spmvb {
namespace bat {
namespace {

// Warps per CTA, columns per copy, slots per warp.  A copy of a whole slice of up
// to 16 columns: with 8 or 4 columns the ring's own instructions cost more than
// copies in flight gain (24 systems of 22,000 rows, us per iteration: 20 warps 16 x
// 1 13.1, 16 x 2 13.4, 8 x 2 14.8; 24 warps 8 x 2 15.2, 4 x 3 21.1).  Two slots of
// 16 would halve the rows a CTA can hold in FP64.
constexpr int OC_NW = 20;
constexpr int OC_U = 16;
constexpr int OC_D = 1;

// The same for one matrix over the grid, whose entries come from memory: more
// warps and copies in flight (us per iteration with nothing kept in L2, 27-point 96^3 / 5-point 1024^2 /
// 7-point 128^3: 28 warps 9 x 2 30.5 / 14.5 / 33.0; 24 warps 9 x 2 30.5 / 15.4 / 36.9;
// 20 warps 9 x 3 30.8 / 15.7 / 40.7, 14 x 2 30.7 / 15.9 / 41.7, 16 x 1 34.5 / 18.3 / 46.2).
constexpr int OCM_NW = 28;
constexpr int OCM_U = 9;
constexpr int OCM_D = 2;

struct OcScalars {
  double rr0, rr_max, rr_true, rr_prev, alpha, beta, s, c;
  int its, refs, status, converged, go, refine, fresh;
};

// The decisions after the sum of A (one thread; every CTA of the group makes
// the same ones from the same totals).  T: the precision alpha is applied in; MX: an
// iteration that breaks down counts (as in the mixed solve's other forms; not in the
// batch's).
template <typename T, bool MX>
__device__ __forceinline__ void oc_step(OcScalars& v, const double (&tot)[4], int kmax,
                                        double rtol2, double delta2) {
  const double rr = tot[3];
  v.refine = 0;
  if (v.its > 0 && !v.fresh) {
    v.rr_max = fmax(v.rr_max, rr);
    v.refine = rr < delta2 * v.rr_max || rr / v.rr0 < rtol2 || v.its >= kmax || !isfinite(rr);
  }
  v.fresh = 0;
  if (v.refine) return;
  const double py = tot[0];
  if (py == 0.0 || !isfinite(py)) {
    v.status = SPMV_ERROR_BREAKDOWN;
    v.go = 0;
    if (MX) v.its += 1;
    return;
  }
  const double al = double(T(rr / py));
  const double rr1 = fmax(rr - 2.0 * al * tot[1] + al * al * tot[2], 0.0);
  v.alpha = al;
  v.beta = rr1 / rr;
  v.rr_prev = rr;
  v.its += 1;
}

// After the sums of R.
__device__ __forceinline__ void oc_refined(OcScalars& v, const double (&tot)[4], int kmax,
                                           double rtol2) {
  v.refs += 1;
  v.rr_true = tot[0];
  v.rr_max = tot[1];
  if (tot[0] / v.rr0 < rtol2) {
    v.converged = 1;
    v.go = 0;
  }
  if (!isfinite(tot[0])) {
    v.status = SPMV_ERROR_BREAKDOWN;
    v.go = 0;
  }
  if (v.its >= kmax) v.go = 0;
  // (beta is 0 where the direction was already restarted: q is then 0.)
  v.s = v.beta > 0.0 ? tot[1] / v.rr_prev / v.beta : 0.0;
  v.c = tot[1] > 0.0 ? tot[2] / tot[1] : 0.0;
  v.fresh = 1;
}

__device__ __forceinline__ float oc_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double oc_fma(double a, double b, double c) {
  return __fma_rn(a, b, c);
}

// A matrix's padding entries (value 0; the batch's have the row's own column).
template <typename CI>
__device__ __forceinline__ bool oc_padding(int c) {
  return sizeof(CI) == 2 ? c == -32768 : c < 0;
}

// The first W columns of a landed slot (vals, idx: the lane's entries): sum += v
// p.  pl: p in shared memory (as the lane's column 0 or, with 16-bit offsets, its
// row), pg: the same place in the unit's p, at row l of the window of `rows`; FULL:
// the window holds every column.
template <int W, bool FULL, bool MX, typename T, typename CI>
__device__ __forceinline__ void oc_slot(const T* vals, const CI* idx, const T* pl, const T* pg,
                                        int l, unsigned rows, T& sum) {
  T x[W];
#pragma unroll
  for (int u = 0; u < W; ++u) {
    const int c = int(idx[32 * u]);
    x[u] = T(0);
    if (!MX || !oc_padding<CI>(c))
      x[u] = FULL || unsigned(l + c) < rows ? pl[c] : __ldcg(pg + c);
  }
#pragma unroll
  for (int u = 0; u < W; ++u) sum = oc_fma(vals[32 * u], x[u], sum);
}
template <int W, bool FULL, bool MX, typename T, typename CI>
__device__ __forceinline__ void oc_slot_of(int w, const T* vals, const CI* idx, const T* pl,
                                           const T* pg, int l, unsigned rows, T& sum) {
  if (w == W)
    oc_slot<W, FULL, MX>(vals, idx, pl, pg, l, rows, sum);
  else if constexpr (W > 1)
    oc_slot_of<W - 1, FULL, MX>(w, vals, idx, pl, pg, l, rows, sum);
}

// ring_pass for this layout, whose entries are all stored ones (padding is the
// row's own column with value 0): no masks, and one code path per number of
// columns.  A pass is bound by the instructions it issues (FP32, 24 systems of
// 22,000 rows of 14 entries: 49 per 32 entries with ring_pass's masks and its test
// of every column against the window).
template <bool FULL, bool MX, typename T, typename CI, int U, int D, class F>
__device__ __forceinline__ bool oc_pass(const RingView<T, CI>& v, RingState& r, const T* ps, int w0,
                                        unsigned rows, const T* pg, F&& f) {
  using Sh = RingShape<T, CI, U, D, 1>;
  const int lane = int(threadIdx.x) & 31;
  int i = 0;
  for (int j = int(threadIdx.x) >> 5; j < v.count; j += v.stride, ++i) {
    const int4 h = v.items[j];
    const int at = h.y - w0 + lane;             // the row in the window
    const int l = sizeof(CI) == 2 ? at : -w0;   // column 0 of the entries
    T sum = T(0);
    int w = h.z & RING_MAX_COLS;
    do {
      if (!mbar_wait_bounded(v.bar + r.rd, (r.phase >> r.rd) & 1u)) return false;
      const unsigned char* slot = v.base + r.rd * Sh::SLOT;
      r.phase ^= 1u << r.rd;
      r.rd = r.rd + 1 == D ? 0 : r.rd + 1;
      oc_slot_of<U, FULL, MX>(min(w, U), reinterpret_cast<const T*>(slot) + lane,
                          reinterpret_cast<const CI*>(slot + Sh::VB) + lane, ps + l, pg + w0 + l, l,
                          rows, sum);
      __syncwarp();
      ring_issue<T, CI, U, D, 1>(v, r);
      w -= U;
    } while (w > 0);
    f(i, at, !MX || lane < (h.z >> 24), sum);
  }
  return true;
}

template <typename T, typename CI, int NW, int U, int D, bool MX>
__global__ void __launch_bounds__(NW * 32, 1) onchip_groups(const __grid_constant__ OnchipArgs a) {
  using Shape = RingShape<T, CI, U, D, 1>;
  using Tm = typename std::conditional<sizeof(T) == 4, Tmem32, Tmem64>::type;
  constexpr int NT = NW * 32;
  constexpr int C = int(sizeof(T)) / 4, CS = 3 * C;  // columns per value, per slice
  extern __shared__ __align__(128) unsigned char oc_smem[];
  __shared__ __align__(8) uint64_t bars[NW * D];
  __shared__ GridTotals<NT, 4> g4;
  __shared__ GridSum<NT> gs;
  __shared__ OcScalars sv;
  __shared__ OnchipCta me;
  __shared__ uint32_t tm_base;
  __shared__ uint64_t policy;
  __shared__ double rr_part[NT];
  const int tid = int(threadIdx.x), warp = tid >> 5, lane = tid & 31;
  int4* const items = reinterpret_cast<int4*>(oc_smem + NW * Shape::BYTES);
  T* const ps = reinterpret_cast<T*>(items + a.per_warp * NW);
  if (tid == 0) {
    me = a.ctas[blockIdx.x];
    policy = a.keep > 0.0f ? l2_policy_part(a.keep) : l2_policy_stream();
  }
  if (lane == 0) ring_init<D>(bars + warp * D);
  if (warp == 0) tmem_alloc(&tm_base, uint32_t(a.alloc));
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  for (int j = tid; j < me.nitems; j += NT) items[j] = __ldg(a.items + me.item0 + j);
  __syncthreads();
  const uint32_t tm =
      tm_base + (uint32_t(warp & 3) << 21) + uint32_t((warp >> 2) * a.per_warp * CS);
  auto view = [&]() {
    return RingView<T, CI>{static_cast<const T*>(a.vals), static_cast<const CI*>(a.idx), items,
                           me.nitems, NW, oc_smem + warp * Shape::BYTES, bars + warp * D,
                           &policy};
  };
  RingState ring;
  ring_prime<T, CI, U, D, 1>(view(), ring);
  const int w0 = me.w0;  // the window's first row
  T* const pg = static_cast<T*>(a.p) + me.vec0;  // the unit's p
  auto each_item = [&](auto&& body) {
    uint32_t t = tm;
    for (int j = warp; j < me.nitems; j += NW, t += CS) body(items[j], items[j].y + lane, t);
  };
  // Whether the lane's row of a slice exists (the batch's rows are padded to whole
  // slices, a matrix's ranks are not).
  auto exists = [&](const int4& h) { return !MX || lane < (h.z >> 24); };
  // The group's syncs, numbered in order; two arrays of partials in turn (a sum
  // may follow another without a barrier between).
  unsigned int epoch = 0;
  auto group_sum = [&](const double(&in)[4], double(&tot)[4]) {
    ++epoch;
    return coop_grid_totals<NT, 4>(in, a.parts + me.part0 + (epoch & 1u) * 4u * unsigned(me.size),
                                   a.bars + me.bar, uint64_t(epoch) * unsigned(me.size), a.err,
                                   a.limit_ns, g4, tot, unsigned(me.rank), unsigned(me.size));
  };
  auto group_barrier = [&]() {
    ++epoch;
    if (me.size == 1) {
      named_sync(1, NT);
      return true;
    }
    return coop_grid_barrier<NT>(a.bars + me.bar, uint64_t(epoch) * unsigned(me.size), a.err,
                                 a.limit_ns, gs);
  };

  // The window's rows of the group's other CTAs, 16 bytes a load (up to 3 of the
  // CTA's own rows at either end come along: the group has them in L2 as well).
  auto load_window = [&]() {
    if (me.size == 1) return;
    constexpr int V = 16 / int(sizeof(T));
    const int before = (me.g0 - w0 + V - 1) / V * V, after = (me.g0 - w0 + me.rows) / V * V;
    const int n = before + me.wrows - after;
#pragma unroll 4
    for (int i = V * tid; i < n; i += V * NT) {
      const int l = i < before ? i : i - before + after;
      *reinterpret_cast<int4*>(ps + l) = __ldcg(reinterpret_cast<const int4*>(pg + w0 + l));
    }
    named_sync(1, NT);
  };

  // Init: r = p = fl(b), x = d = 0.
  double tot[4], rr = 0.0;
  {
    double in[4] = {0.0, 0.0, 0.0, 0.0};
    each_item([&](const int4& h, int g, uint32_t t) {
      double bi = 0.0;
      if (MX) {
        if (exists(h)) bi = a.b[g];
      } else {
        const int pr = a.perm[me.perm0 + g];
        if (pr >= 0)
          bi = me.col < 0 ? a.b_user[me.sys][pr] : a.B_user[int64_t(pr) * a.nrhs + me.col];
        a.b[me.vec0 + g] = bi;
      }
      const T ri = T(bi);
      if (exists(h)) {
        __stcg(a.x + me.vec0 + g, 0.0);
        ps[g - w0] = ri;
        if (me.size > 1) __stcg(pg + g, ri);
      }
      in[0] += bi * bi;
      rr += double(ri) * double(ri);
      __syncwarp();
      tmem_st(t, ri);
      tmem_st(t + 2 * C, T(0));
    });
    __syncwarp();
    tmem_wait_st();
    in[1] = rr;
    rr_part[tid] = rr;
    // Every unit has read its right-hand side before any unit's solution is
    // written (the caller may pass one buffer as both).
    const bool all = MX || coop_grid_barrier<NT>(a.bars, gridDim.x, a.err, a.limit_ns, gs);
    const bool ok = all && group_sum(in, tot);
    if (tid == 0) {
      sv = OcScalars{};
      sv.status = SPMV_SUCCESS;
      if (ok) {
        sv.rr0 = sv.rr_true = tot[0];
        sv.rr_max = tot[1];
        sv.converged = tot[0] == 0.0;
        sv.go = a.kmax > 0 && tot[0] > 0.0 && isfinite(tot[0]);
      }
      gs.ok = ok;
    }
    named_sync(1, NT);
  }
  bool ok = gs.ok != 0;
  while (sv.go) {
    // A: y = A p and the four sums.
    {
      double in[4] = {0.0, 0.0, 0.0, rr_part[tid]};
      load_window();
      const unsigned rows = unsigned(me.wrows);
      auto row_sums = [&](int i, int at, bool row, T y) {
        const uint32_t t = tm + i * CS;
        Tm rv;
        __syncwarp();
        tmem_ld(t, rv);
        tmem_st(t + C, y);
        tmem_wait_ld(rv);
        const double yd = double(y);  // (a lane without a row: r and y are 0, p is not its own)
        in[0] += double(row ? ps[at] : T(0)) * yd;
        in[1] += double(rv.get()) * yd;
        in[2] += yd * yd;
      };
      if (!(me.full
                ? oc_pass<true, MX, T, CI, U, D>(view(), ring, ps, w0, rows, pg, row_sums)
                : oc_pass<false, MX, T, CI, U, D>(view(), ring, ps, w0, rows, pg, row_sums)))
        if (lane == 0) atomicExch(a.err, 1);
      __syncwarp();
      tmem_wait_st();
      if (!(ok = group_sum(in, tot))) break;
      if (tid == 0) oc_step<T, MX>(sv, tot, a.kmax, a.rtol2, a.delta2);
      named_sync(1, NT);
    }
    if (!sv.go) break;
    rr = 0.0;
    if (!sv.refine) {
      // C, two slices in flight per warp.
      const T alpha = T(sv.alpha), beta = T(sv.beta);
      const int n = me.nitems;
      auto update = [&](auto count, int j, uint32_t t) {
        constexpr int B = decltype(count)::value;
        int4 h[B];
        int l[B];
        T pv[B];
        Tm r[B], y[B], d[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
          h[b] = items[j + b * NW];
          l[b] = h[b].y - w0 + lane;
          pv[b] = ps[l[b]];
        }
        __syncwarp();
#pragma unroll
        for (int b = 0; b < B; ++b) {
          tmem_ld(t + b * CS, r[b]);
          tmem_ld(t + b * CS + C, y[b]);
          tmem_ld(t + b * CS + 2 * C, d[b]);
        }
        tmem_wait_ld(r, y, d);
#pragma unroll
        for (int b = 0; b < B; ++b) {
          const T rn = r[b].get() - alpha * y[b].get(), pn = rn + beta * pv[b];
          __syncwarp();
          tmem_st(t + b * CS, rn);
          tmem_st(t + b * CS + 2 * C, d[b].get() + alpha * pv[b]);
          if (exists(h[b])) {
            ps[l[b]] = pn;
            if (me.size > 1) __stcg(pg + w0 + l[b], pn);
          }
          rr += double(rn) * double(rn);
        }
      };
      uint32_t t = tm;
      for (int j = warp; j < n; j += 2 * NW, t += 2 * CS) {
        if (j + NW < n)
          update(std::integral_constant<int, 2>{}, j, t);
        else
          update(std::integral_constant<int, 1>{}, j, t);
      }
      __syncwarp();
      tmem_wait_st();
      rr_part[tid] = rr;
      if (!(ok = group_barrier())) break;
      continue;
    }
    // R: x += d, d = 0.
    each_item([&](const int4& h, int g, uint32_t t) {
      Tm dv;
      __syncwarp();
      tmem_ld(t + 2 * C, dv);
      tmem_wait_ld(dv);
      double* const xp = a.x + me.vec0 + g;
      if (exists(h)) __stcg(xp, __ldcg(xp) + double(dv.get()));
      __syncwarp();
      tmem_st(t + 2 * C, T(0));
    });
    __syncwarp();
    tmem_wait_st();
    if (!(ok = group_barrier())) break;
    // r = fl(b - A64 x), q in y's place.
    {
      double in[4] = {0.0, 0.0, 0.0, 0.0};
      const CI* const idx = static_cast<const CI*>(a.idx);
      const double* const xu = a.x + me.vec0;
      each_item([&](const int4& h, int g, uint32_t t) {
        const int w = h.z & RING_MAX_COLS;
        const int64_t e = int64_t(h.x) * 32 + lane;
        double acc = 0.0;
        for (int k = 0; k < w; k += 4) {
          double v[4], xv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const bool in_row = k + u < w;
            const int64_t at = e + 32 * int64_t(in_row ? k + u : k);
            const int ci = int(idx[at]);
            v[u] = in_row ? a.vals64[at] : 0.0;
            xv[u] = 0.0;
            if (!MX || !oc_padding<CI>(ci)) xv[u] = __ldcg(xu + (sizeof(CI) == 2 ? g + ci : ci));
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (k + u < w) acc += v[u] * xv[u];
        }
        const double r64 = exists(h) ? a.b[me.vec0 + g] - acc : 0.0;
        const T rn = T(r64);
        Tm rv;
        __syncwarp();
        tmem_ld(t, rv);
        tmem_wait_ld(rv);
        const T q = exists(h) ? ps[g - w0] - rv.get() : T(0);
        __syncwarp();
        tmem_st(t, rn);
        tmem_st(t + C, q);
        in[0] += r64 * r64;
        in[1] += double(rn) * double(rn);
        in[2] += double(rn) * double(q);
      });
      __syncwarp();
      tmem_wait_st();
      rr_part[tid] = in[1];
      if (!(ok = group_sum(in, tot))) break;
      if (tid == 0) oc_refined(sv, tot, a.kmax, a.rtol2);
      named_sync(1, NT);
    }
    if (!sv.go) break;
    {
      const T s = T(sv.s), c = T(sv.c);
      each_item([&](const int4& h, int g, uint32_t t) {
        Tm rv, qv;
        __syncwarp();
        tmem_ld(t, rv);
        tmem_ld(t + C, qv);
        tmem_wait_ld(rv, qv);
        const T pn = rv.get() + s * (qv.get() - c * rv.get());
        if (exists(h)) {
          ps[g - w0] = pn;
          if (me.size > 1) __stcg(pg + g, pn);
        }
        __syncwarp();
      });
    }
    if (!(ok = group_barrier())) break;
  }
  if (ok) {
    each_item([&](const int4& h, int g, uint32_t t) {
      Tm dv;
      __syncwarp();
      tmem_ld(t + 2 * C, dv);
      tmem_wait_ld(dv);
      const int pr = MX ? -1 : a.perm[me.perm0 + g];
      const double xi = exists(h) ? __ldcg(a.x + me.vec0 + g) + double(dv.get()) : 0.0;
      if (MX) {
        if (exists(h)) a.x[g] = xi;
      } else if (pr >= 0) {
        if (me.col < 0)
          a.x_user[me.sys][pr] = xi;
        else
          a.X_user[int64_t(pr) * a.nrhs + me.col] = xi;
      }
      __syncwarp();
    });
    if (tid == 0 && me.rank == 0) {
      Slot o{};
      o.rr0 = sv.rr0;
      o.rr_true = sv.rr_true;
      o.its = sv.its;
      o.refs = sv.refs;
      o.status = sv.status;
      o.converged = sv.converged;
      a.slots[me.slot] = o;
    }
  }
  ring_drain<T, CI, D>(view(), ring);
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0) tmem_free(tm_base, uint32_t(a.alloc));
}

// Smallest and largest column of each slice of a matrix (its first row, where it
// has no entry).
template <typename CI>
__global__ void __launch_bounds__(256) oc_bounds(const int4* __restrict__ items, int n,
                                                 const CI* __restrict__ idx,
                                                 int2* __restrict__ out) {
  const int i = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = int(threadIdx.x) & 31;
  if (i >= n) return;
  const int4 h = items[i];
  const int w = h.z & RING_MAX_COLS;
  int lo = h.y, hi = h.y;
  for (int k = 0; k < w; ++k) {
    const int c = int(idx[(int64_t(h.x) + k) * 32 + lane]);
    if (oc_padding<CI>(c)) continue;
    const int col = sizeof(CI) == 2 ? h.y + lane + c : c;
    lo = min(lo, col);
    hi = max(hi, col);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0) out[i] = make_int2(lo, hi);
}

struct OcKernel {
  const void* fn;
  int64_t ring_bytes;
};
template <typename T, typename CI>
OcKernel oc_kernel() {
  return {(const void*)onchip_groups<T, CI, OC_NW, OC_U, OC_D, false>,
          OC_NW * int64_t(RingShape<T, CI, OC_U, OC_D, 1>::BYTES)};
}
template <typename CI>
OcKernel ocm_kernel() {
  return {(const void*)onchip_groups<float, CI, OCM_NW, OCM_U, OCM_D, true>,
          OCM_NW * int64_t(RingShape<float, CI, OCM_U, OCM_D, 1>::BYTES)};
}
OcKernel oc_kernel(bool fp32, bool d16) {
  if (fp32) return d16 ? oc_kernel<float, int16_t>() : oc_kernel<float, int32_t>();
  return d16 ? oc_kernel<double, int16_t>() : oc_kernel<double, int32_t>();
}

// Estimated cost of a unit's solve over c CTAs: microseconds per iteration (the
// busiest warp's slices, 1.16 each at 14 entries per row, and the rest, 3.6 with one
// CTA and 6.1 with others to wait for), times the iterations, which grow with the
// rows (mesh systems: 181 at 2,048, 315 at 24,000, about the fifth root; without
// that factor the batch above takes 3.7 ms for 3.5).
double oc_cost(int64_t slices, double width, int64_t c) {
  const int64_t per_cta = (slices + c - 1) / c, items = (per_cta + OC_NW - 1) / OC_NW;
  const double us = double(items) * (0.25 + 0.065 * width) + (c > 1 ? 6.1 : 3.6);
  return us * std::pow(double(slices), 0.2);
}

// Windows that do not fit in `fit` rows are cut down to the CTA's own rows;
// returns the rows of the largest.
int64_t fit_windows(OnchipPlan& p, int64_t fit) {
  int64_t rows = 0;
  for (OnchipCta& c : p.ctas) {
    c.full = c.wrows <= fit;
    if (!c.full) {
      c.wrows = (c.rows + c.g0 - c.g0 / 4 * 4 + 3) / 4 * 4;
      c.w0 = c.g0 / 4 * 4;
    }
    rows = std::max<int64_t>(rows, c.wrows);
  }
  return rows;
}

}  // namespace

bool plan_onchip_matrix(spmv_matrix A, OnchipPlan& out) {
  out = OnchipPlan{};
  const bool d16 = A->fwd.d16;
  const OcKernel kn = d16 ? ocm_kernel<int16_t>() : ocm_kernel<int32_t>();
  out.fn = kn.fn;
  out.block = OCM_NW * 32;
  const ItemTable& t = item_table(A, 1);
  if (!t.ok) return false;
  const spmv_comm comm = A->comm;
  const int n = t.nitems, grid = std::max(1, std::min(comm->num_sms, n));
  std::vector<int2> bound;
  bound.resize(size_t(n));
  DevBuf db;
  db.reserve(sizeof(int2) * size_t(n));
  const int blocks = (n + 7) / 8;
  if (d16)
    oc_bounds<int16_t><<<blocks, 256, 0, comm->stream>>>(
        t.desc.as<int4>(), n, A->fwd.sell_d16_global.as<int16_t>(), db.as<int2>());
  else
    oc_bounds<int32_t><<<blocks, 256, 0, comm->stream>>>(
        t.desc.as<int4>(), n, A->fwd.sell_cols_global.as<int32_t>(), db.as<int2>());
  SPMVB_CUDA(cudaGetLastError());
  SPMVB_CUDA(cudaMemcpyAsync(bound.data(), db.ptr, sizeof(int2) * size_t(n),
                             cudaMemcpyDeviceToHost, comm->stream));
  SPMVB_CUDA(cudaStreamSynchronize(comm->stream));
  int64_t most = 0, own = 0;
  for (int b = 0; b < grid; ++b) {
    const int a0 = int(int64_t(n) * b / grid), a1 = int(int64_t(n) * (b + 1) / grid);
    OnchipCta c{};
    c.item0 = a0;
    c.nitems = a1 - a0;
    c.g0 = t.row[size_t(a0)];
    c.rows = t.row[size_t(a1)] - c.g0;
    int lo = c.g0, hi = c.g0 + c.rows;
    for (int k = a0; k < a1; ++k) {
      lo = std::min(lo, bound[size_t(k)].x);
      hi = std::max(hi, bound[size_t(k)].y + 1);
    }
    c.w0 = lo / 4 * 4;
    c.wrows = (hi - c.w0 + 3) / 4 * 4;
    c.bar = 0;
    c.rank = b;
    c.size = grid;
    out.ctas.push_back(c);
    most = std::max<int64_t>(most, a1 - a0);
    own = std::max<int64_t>(own, c.rows + 8);
  }
  out.parts = 8 * int64_t(grid);
  out.per_warp = int((most + OCM_NW - 1) / OCM_NW);
  const int cols = out.per_warp * (OCM_NW / 4) * 3;
  if (cols > 512) return false;
  out.alloc = 32;
  while (out.alloc < cols) out.alloc *= 2;
  // (32 rows more: lanes without a row read past the last one.)
  const int64_t fixed = kn.ring_bytes + int64_t(out.per_warp) * OCM_NW * int64_t(sizeof(int4)) +
                        32 * int64_t(sizeof(float));
  const int64_t most_smem = allow_dynamic_smem(kn.fn, comm->device);
  if (fixed + 4 * own > most_smem) return false;
  out.smem = fixed + 4 * fit_windows(out, (most_smem - fixed) / 4);
  int nb = 0;
  SPMVB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kn.fn, out.block,
                                                           size_t(out.smem)));
  out.ok = nb >= 1;
  return out.ok;
}

bool plan_onchip(const Plan& P, int block_sys, int nrhs, bool fp32, int device, int num_sms,
                 OnchipPlan& out) {
  const int vb = fp32 ? 4 : 8;
  const OcKernel kn = oc_kernel(fp32, P.fits16);
  out = OnchipPlan{};
  out.fn = kn.fn;
  out.block = OC_NW * 32;
  if (P.entries / 32 > int64_t(INT32_MAX) || P.max_width > RING_MAX_COLS) return false;
  struct U {
    int sys, col, ctas;
    int64_t slices;
    double width, cost;
  };
  std::vector<U> units;
  auto add = [&](int sys, int col) {
    if (P.n[sys] == 0) return;
    U u{};
    u.sys = sys;
    u.col = col;
    u.slices = (P.n[sys] + 31) / 32;
    u.width = double(P.sys_entries[sys]) / (32.0 * double(u.slices));
    units.push_back(u);
  };
  for (int i = 0; i < P.nsys; ++i) add(i, -1);
  for (int l = 0; l < nrhs; ++l) add(block_sys, l);
  if (units.empty() || int(units.size()) > num_sms) return false;
  // Slices a CTA can hold: tensor memory's 512 columns, shared memory.
  const int cols = 3 * vb / 4;
  auto smem_of = [&](int per_warp, int64_t rows) {
    return kn.ring_bytes + int64_t(per_warp) * OC_NW * int64_t(sizeof(int4)) + rows * vb;
  };
  const int64_t most_smem = allow_dynamic_smem(kn.fn, device);
  int per_warp = 512 / (OC_NW / 4 * cols);
  while (per_warp > 0 && smem_of(per_warp, 32 * per_warp * OC_NW) > most_smem) --per_warp;
  if (per_warp == 0) return false;
  const int64_t cap = int64_t(per_warp) * OC_NW;
  // One CTA each, or as many as the unit's rows need; the rest to whichever
  // unit is estimated slowest, as long as that helps it.
  int64_t left = num_sms;
  auto slower = [](const U* x, const U* y) { return x->cost < y->cost; };
  std::priority_queue<U*, std::vector<U*>, decltype(slower)> queue(slower);
  for (U& u : units) {
    u.ctas = int((u.slices + cap - 1) / cap);
    u.cost = oc_cost(u.slices, u.width, u.ctas);
    left -= u.ctas;
    queue.push(&u);
  }
  if (left < 0) return false;
  while (!queue.empty()) {
    U* u = queue.top();
    queue.pop();
    // The next counts with fewer items in the busiest warp; the first that is
    // faster by the estimate.
    for (int64_t items = ((u->slices + u->ctas - 1) / u->ctas + OC_NW - 1) / OC_NW - 1; items > 0;
         --items) {
      const int64_t c = (u->slices + items * OC_NW - 1) / (items * OC_NW);
      if (c - u->ctas > left) break;
      const double cost = oc_cost(u->slices, u->width, c);
      if (cost >= u->cost) continue;
      left -= c - u->ctas;
      u->ctas = int(c);
      u->cost = cost;
      queue.push(u);
      break;
    }
  }
  int64_t rows = 0, parts = 0, most = 0;
  int bar = 1;
  for (const U& u : units) {
    const int64_t s0 = P.slice0[u.sys];
    for (int r = 0; r < u.ctas; ++r) {
      OnchipCta c{};
      const int64_t a0 = u.slices * r / u.ctas, a1 = u.slices * (r + 1) / u.ctas;
      c.item0 = s0 + a0;
      c.nitems = int(a1 - a0);
      c.g0 = int(32 * a0);
      c.rows = int(32 * (a1 - a0));
      int lo = int(32 * a0), hi = int(32 * a1);
      for (int64_t k = s0 + a0; k < s0 + a1; ++k) {
        lo = std::min(lo, P.sbound[size_t(2 * k)] & ~31);
        hi = std::max(hi, (P.sbound[size_t(2 * k + 1)] | 31) + 1);
      }
      c.w0 = lo;
      c.wrows = hi - lo;
      c.vec0 = rows;
      c.perm0 = P.row0[u.sys];
      c.part0 = parts;
      c.bar = bar * OC_BAR;
      c.rank = r;
      c.size = u.ctas;
      c.sys = u.sys;
      c.col = u.col;
      c.slot = u.col < 0 ? u.sys : P.nsys + u.col;
      out.ctas.push_back(c);
      most = std::max(most, a1 - a0);
    }
    rows += 32 * u.slices;
    parts += 8 * int64_t(u.ctas);
    ++bar;
  }
  out.rows = rows;
  out.parts = parts;
  out.nbars = bar;
  out.per_warp = int((most + OC_NW - 1) / OC_NW);
  out.alloc = 32;
  while (out.alloc < out.per_warp * (OC_NW / 4) * cols) out.alloc *= 2;
  const int64_t wrows = fit_windows(out, (most_smem - smem_of(out.per_warp, 0)) / vb);
  out.smem = smem_of(out.per_warp, wrows);
  int nb = 0;
  SPMVB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kn.fn, OC_NW * 32,
                                                           size_t(out.smem)));
  out.ok = nb >= 1;
  return out.ok;
}

bool launch_onchip(const OnchipPlan& plan, OnchipArgs& a, cudaStream_t s) {
  void* args[] = {&a};
  const cudaError_t e =
      cudaLaunchCooperativeKernel(plan.fn, dim3(unsigned(plan.ctas.size())), dim3(unsigned(plan.block)),
                                  args, size_t(plan.smem), s);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    (void)cudaGetLastError();
    return false;
  }
  SPMVB_CUDA(e);
  return true;
}

}  // namespace bat
}  // namespace spmvb
