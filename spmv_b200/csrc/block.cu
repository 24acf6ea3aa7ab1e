// Multi-right-hand-side product and block CG (no counterpart in the
// reference; builds on Matrix::operator* and spmv::cg, cg.cpp:11-83).
//
// Vectors of k right-hand sides are stored row-major (n x k, leading
// dimension k), so the k values of one row are contiguous.  A row is computed
// by a group of KL lanes, each with a run of right-hand sides (Run below:
// 16-byte accesses of X and Y where k and the vectors' alignment allow); every
// lane of the group reads the row's columns and values (one broadcast
// transaction).  A is read once for all k right-hand sides.
//
// What bounds the product: X is gathered from L2, 8 k bytes per entry, behind
// a chain of dependent loads (row pointer, column, X).  So each lane keeps
// SPMM_BATCH entries in flight and issues every batch whole (a tail of single
// entries costs one chain each), the next row's pointers are loaded a row
// ahead, and a CTA takes a chunk of neighbouring rows.  Rows longer
// than LONG_ROW entries are left to the whole CTA.  Against one right-hand
// side per lane, batches of four and a tail (FP64, 7-point 96^3, 4 ranks):
// k = 2 24.7 -> 20.2 us, k = 8 69.8 -> 59.3, k = 16 133 -> 104 (3.0 TB/s of
// compulsory traffic), k = 32 250 -> 189; with rows of up to 12,500 entries
// (100,003 power-law rows, k = 8) 1.38 ms -> 70 us.
//
// Block CG runs k independent CG recurrences that share each product: the
// SpMM's epilogue forms the k dot products p_l . (A p)_l, and every column has
// its own alpha, beta, convergence test (cg.cpp:78) and breakdown flag; a
// converged column stops changing.  The loop ends when every column has
// converged or broken down, or after max_its iterations.  A solve is one
// cooperative launch of persistent CTAs (one per SM: grid sums cost more with
// every CTA that takes part; k = 2 on 250k rows, 24 us per iteration with three
// CTAs of 256 threads per SM, 19 with one of 1024) with two grid sums of k
// values and one grid barrier per iteration, the same form as the fused single
// solve (cg.cu).  Its workspace is kept with the matrix.  Per iteration on
// 64 x 64 x 61, 4 ranks: k = 1 17.8 us, k = 8 39, k = 32 160; as a CUDA graph
// of three kernels whose column sums one thread added over the grid, 120-160,
// 217 and 425.
#include <algorithm>
#include <cmath>

#include "internal.h"
#include "spmv_kernel.cuh"

struct BlockWorkspace {
  int64_t n = 0;
  // b, x, r, p, y (n x k, for the largest k solved so far), per-CTA partials,
  // state and the grid barrier's counter.
  spmvb::DevBuf b, x, r, p, y, partials, state;
  std::vector<spmvb::DevBuf*> vectors() { return {&b, &x, &r, &p, &y}; }
};

namespace spmvb {

namespace {

constexpr int BBS = 256;       // threads per CTA
constexpr int BCPS = 4;            // CTAs per SM the block product is compiled to fit
constexpr int CBS = 1024;          // threads per CTA of block CG, one CTA per SM
constexpr int MAXK = 32;
constexpr int SPMM_BATCH = 8;      // entries in flight per lane
constexpr int LONG_ROW = 512;      // entries above which a row is the whole CTA's
// Values of X per chunk of rows: the product's chunks keep their X rows and
// their neighbours' in L1; the solver's are one per CTA up to this size (its
// vectors then stay in L2 between the phases).
constexpr int SPMM_CHUNK = 4096, BCG_CHUNK = 24576;
// Bytes of vectors a matrix keeps between block solves.  (Allocating and freeing them
// takes 3 ms for 0.67 GB, 128^3 rows and k = 8, where 40 iterations take 15, and 5.4 ms
// for 2.7 GB, k = 32, where they take 52.)
constexpr size_t BCG_KEEP = size_t(1) << 30;

// Right-hand sides per lane.  V consecutive ones, the vectors aligned to V
// values (SPLIT false); or two, loaded one by one, the second missing from
// the last lane of an odd k (SPLIT).
template <int V_, bool SPLIT_>
struct Run {
  static constexpr int V = V_;
  static constexpr bool SPLIT = SPLIT_;
  int c0;    // first right-hand side
  int next;  // SPLIT: offset of the second (0 when there is none)
  bool on;
  __device__ __forceinline__ Run(int member, int k)
      : c0(member * V), next(member * V + 1 < k ? 1 : 0), on(member * V < k) {}
};

template <typename T, class R>
__device__ __forceinline__ void ld_run(const R& r, const T* p, T (&o)[R::V]) {
  if constexpr (R::V == 1) {
    o[0] = *p;
  } else if constexpr (R::SPLIT) {
    o[0] = p[0];
    o[1] = p[r.next];
  } else if constexpr (sizeof(T) * R::V == 16) {
    const typename VecT<T>::V t = *reinterpret_cast<const typename VecT<T>::V*>(p);
#pragma unroll
    for (int i = 0; i < R::V; ++i) o[i] = comp(t, i);
  } else {
    const float2 t = *reinterpret_cast<const float2*>(p);
    o[0] = t.x;
    o[1] = t.y;
  }
}
template <typename T, class R>
__device__ __forceinline__ void st_run(const R& r, T* p, const T (&v)[R::V]) {
  if constexpr (R::V == 1) {
    *p = v[0];
  } else if constexpr (R::SPLIT) {
    p[0] = v[0];
    if (r.next) p[1] = v[1];
  } else if constexpr (sizeof(T) == 8) {
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
  } else if constexpr (R::V == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  }
}

// acc += the row's entries below e from j on, in batches of SPMM_BATCH
// consecutive entries at j, j + step, ...  Every batch is issued whole: past
// the end it repeats the last entry and the sum skips it.  (X may be written
// between the calls of one launch, so it is read with ordinary loads.)
template <typename T, class R>
__device__ __forceinline__ void spmm_entries(const R& r, const int32_t* cols, const T* vals,
                                             const T* xc, int k, int j, int e, int step,
                                             T (&acc)[R::V]) {
  constexpr int BU = SPMM_BATCH;
  for (; j < e; j += step) {
    int c[BU];
    T v[BU], xv[BU][R::V];
#pragma unroll
    for (int u = 0; u < BU; ++u) c[u] = __ldg(cols + min(j + u, e - 1));
#pragma unroll
    for (int u = 0; u < BU; ++u) ld_run<T>(r, xc + int64_t(c[u]) * k, xv[u]);
#pragma unroll
    for (int u = 0; u < BU; ++u) v[u] = __ldg(vals + min(j + u, e - 1));
#pragma unroll
    for (int u = 0; u < BU; ++u)
      if (j + u < e)
#pragma unroll
        for (int i = 0; i < R::V; ++i) acc[i] += v[u] * xv[u][i];
  }
}

// Rows [lo, hi) of a rank's Y = A X, by the whole CTA, KL lanes per row: f(P, row, run,
// sums) once per row and lane that has right-hand sides.
template <typename T, int NT, int KL, class R, class F>
__device__ __forceinline__ void spmm_rows(const PartArg& P, int k, int lo, int hi, F&& f) {
  constexpr int V = R::V;
  __shared__ T group_sums[NT * V];
  __shared__ unsigned int long_mask[NT / 32];
  const int tid = int(threadIdx.x), grp = tid / KL;
  const R run(tid % KL, k);
  const T* xc = static_cast<const T*>(P.x) + (run.on ? run.c0 : 0);
  const T* vals = static_cast<const T*>(P.vals);
  int row = lo + grp;
  int s = 0, e = 0, any_long = 0;
  if (row < hi) {
    s = __ldg(P.rowptr + row);
    e = __ldg(P.rowptr + row + 1);
  }
  while (row < hi) {
    const int next = row + NT / KL;
    int sn = 0, en = 0;
    if (next < hi) {
      sn = __ldg(P.rowptr + next);
      en = __ldg(P.rowptr + next + 1);
    }
    if (e - s > LONG_ROW) {
      any_long = 1;
    } else {
      T acc[V];
#pragma unroll
      for (int i = 0; i < V; ++i) acc[i] = T(0);
      spmm_entries<T>(run, P.cols, vals, xc, k, s, e, SPMM_BATCH, acc);
      if (run.on) f(P, row, run, acc);
    }
    row = next;
    s = sn;
    e = en;
  }
  if (!__syncthreads_or(any_long)) return;
  // Long rows, in row order: every group takes batches in
  // turn; the groups' sums are added in group order.
  for (int r0 = lo; r0 < hi; r0 += NT) {
    const int mine = r0 + tid;
    const bool is_long =
        mine < hi && __ldg(P.rowptr + mine + 1) - __ldg(P.rowptr + mine) > LONG_ROW;
    const unsigned int m = __ballot_sync(0xffffffffu, is_long);
    if ((tid & 31) == 0) long_mask[tid >> 5] = m;
    __syncthreads();
    for (int w = 0; w < NT / 32; ++w)
      for (unsigned int left = long_mask[w]; left != 0; left &= left - 1) {
        const int lrow = r0 + 32 * w + __ffs(left) - 1;
        const int ls = __ldg(P.rowptr + lrow), le = __ldg(P.rowptr + lrow + 1);
        T acc[V];
#pragma unroll
        for (int i = 0; i < V; ++i) acc[i] = T(0);
        spmm_entries<T>(run, P.cols, vals, xc, k, ls + grp * SPMM_BATCH, le,
                        SPMM_BATCH * (NT / KL), acc);
#pragma unroll
        for (int i = 0; i < V; ++i) group_sums[tid * V + i] = acc[i];
        __syncthreads();
        if (grp == 0 && run.on) {
#pragma unroll
          for (int i = 0; i < V; ++i) {
            T t = T(0);
            for (int g = 0; g < NT / KL; ++g) t += group_sums[g * KL * V + run.c0 + i];
            acc[i] = t;
          }
          f(P, lrow, run, acc);
        }
        __syncthreads();
      }
    __syncthreads();
  }
}

// Each CTA a chunk of `rows` rows of one rank, which it finds by bisection.  (Chunks
// across the ranks' borders, found by passing the ranks in turn, cost small products 1 to
// 2 us of latency: every rank is a constant line of its own, and a chunk over a border
// takes two passes that all others wait for.  FP64, 8,000 7-point rows over 8 ranks, k = 8
// 6.2 us, now 4.1 to 5; 884,736 rows over 4 ranks, k = 8 59.4 and 55.6, k = 32 195 and
// 178.)
template <typename T, int KL, class R>
__global__ void __launch_bounds__(BBS, BCPS)
    spmm_kernel(const __grid_constant__ SpmvArgs a, int rows, int k) {
  const PartArg& P = a.part[find_part(a, blockIdx.x)];
  const int lo = (int(blockIdx.x) - P.block_begin) * rows;
  const int hi = P.nrows - lo < rows ? P.nrows : lo + rows;
  if (lo >= hi) return;
  spmm_rows<T, BBS, KL, R>(P, k, lo, hi,
                           [&](const PartArg& P, int row, const R& run, const T(&acc)[R::V]) {
                             st_run<T>(run, static_cast<T*>(P.y) + int64_t(row) * k + run.c0,
                                       acc);
                           });
}

// One right-hand side per lane, KL lanes per row, CTAs striding over tiles of
// BBS / KL rows; batches of four entries and a tail of single ones, in 32
// registers (every warp slot of the SM taken).  For products whose lanes cannot
// load aligned runs of X, and whose rows either take several batches of
// spmm_kernel or leave most of one empty (use_walk).
template <typename T, int KL>
__global__ void __launch_bounds__(BBS)
    spmm_walk_kernel(const __grid_constant__ SpmvArgs a, int k) {
  const int p = find_part(a, blockIdx.x);
  const PartArg& P = a.part[p];
  const int32_t* __restrict__ cols = P.cols;
  const T* __restrict__ vals = static_cast<const T*>(P.vals);
  const T* __restrict__ x = static_cast<const T*>(P.x);
  const int group = int(threadIdx.x) / KL, lane = int(threadIdx.x) % KL;
  const bool on = lane < k;
  for (int tile = int(blockIdx.x) - P.block_begin; tile < P.ntiles; tile += P.nblocks) {
    const int row = tile * (BBS / KL) + group;
    if (row >= P.nrows) continue;
    const int s = __ldg(P.rowptr + row), e = __ldg(P.rowptr + row + 1);
    T acc = T(0);
    int j = s;
    for (; j + 4 <= e; j += 4) {
      int c[4];
      T v[4], xv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        c[u] = __ldg(cols + j + u);
        v[u] = __ldg(vals + j + u);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) xv[u] = on ? __ldg(x + int64_t(c[u]) * k + lane) : T(0);
#pragma unroll
      for (int u = 0; u < 4; ++u) acc += v[u] * xv[u];
    }
    for (; j < e; ++j) {
      const int c = __ldg(cols + j);
      const T v = __ldg(vals + j);
      if (on) acc += v * __ldg(x + int64_t(c) * k + lane);
    }
    if (on) static_cast<T*>(P.y)[int64_t(row) * k + lane] = acc;
  }
}

// ---------------------------------------------------------------------------
// Block CG
// ---------------------------------------------------------------------------
// The rows of all ranks in equal chunks of consecutive rows (global numbering): chunk q
// is [q rows, (q + 1) rows).
struct RowChunks {
  int64_t rows, total;  // rows per chunk, rows in all
  int count;
  __host__ __device__ int64_t begin(int64_t q) const { return q * rows; }
  __host__ __device__ int64_t end(int64_t q) const {
    return (q + 1) * rows < total ? (q + 1) * rows : total;
  }
};

// g(P, lo, hi) for each rank's rows among [g0, g1) (global numbering).
template <class G>
__device__ __forceinline__ void each_rank(const SpmvArgs& a, int64_t g0, int64_t g1, G&& g) {
  int64_t row0 = 0;
  for (int p = 0; p < a.nparts; ++p) {
    const PartArg& P = a.part[p];
    const int64_t first = row0;
    row0 += P.nrows;
    const int lo = int(max(g0, first) - first), hi = int(min(g1, row0) - first);
    if (g0 >= row0 || g1 <= first || lo >= hi) continue;
    g(P, lo, hi);
  }
}

struct BcgState {
  double rr0[MAXK], rr[MAXK];
  int status[MAXK], its[MAXK];
  unsigned long long bar;
  int err, pad;
};

struct BcgPtrs {
  const double* b;
  double* x;
  double* r;
  double* p;
  double* y;
  double* partials;  // two arrays of [CTAs][MAXK]
  BcgState* st;
  int nrhs, kmax;
  double rtol2;
  unsigned long long wait_ns;
};

struct BcgShared {
  double red[CBS * 2];          // per-thread sums, V per thread
  double part[CBS / 32][MAXK];  // per-warp sums of the partials
  double tot[MAXK];
  double rr0[MAXK], rr[MAXK], alpha[MAXK], beta[MAXK];
  int active[MAXK], status[MAXK], its[MAXK];
  int ok;
};

// Sum over the grid of every column's share: thread t holds V sums of columns
// (t % stride) V .. + V - 1 (threads from `used` on hold none).  All threads
// of every CTA get the totals in sh.tot, in the same fixed order: a CTA adds
// its threads in index order by 32 lanes per column, publishes one partial
// per column, and after the barrier every CTA adds all partials.
template <int V>
__device__ __forceinline__ bool column_sums(const double (&v)[V], int stride, int used,
                                            const BcgPtrs& c, double* parts,
                                            unsigned long long target, BcgShared& sh) {
  const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int i = 0; i < V; ++i) sh.red[tid * V + i] = v[i];
  __syncthreads();
  for (int col = warp; col < c.nrhs; col += CBS / 32) {
    double t = 0.0;
    for (int q = col / V + lane * stride; q < used; q += 32 * stride)
      t += sh.red[q * V + col % V];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) __stcg(parts + blockIdx.x * MAXK + col, t);
  }
  __syncthreads();
  if (tid == 0) sh.ok = grid_arrive_wait(&c.st->bar, target, &c.st->err, c.wait_ns);
  __syncthreads();
  if (!sh.ok) return false;
  double t = 0.0;
  if (lane < c.nrhs)
    for (unsigned int b = warp; b < gridDim.x; b += CBS / 32) t += __ldcg(parts + b * MAXK + lane);
  sh.part[warp][lane] = t;
  __syncthreads();
  if (tid < c.nrhs) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < CBS / 32; ++w) s += sh.part[w][tid];
    sh.tot[tid] = s;
  }
  __syncthreads();
  return true;
}

// One cooperative launch per solve.  Per iteration, on the CTA's rows:
//   A  Y = A P, p.y                                  -> grid sum, alpha
//   B  r -= alpha y, r.r                             -> grid sum, beta, tests
//   C  x += alpha p, p = r + beta p                  -> grid barrier
// (columns that have stopped are left as they are).
template <int KL, class R>
__global__ void __launch_bounds__(CBS)
    bcg_kernel(const __grid_constant__ SpmvArgs a, const BcgPtrs c,
               const RowChunks ch) {
  // Right-hand sides per thread in the vector phases.
  constexpr int V = R::SPLIT ? 1 : R::V;
  using RV = Run<V, false>;
  __shared__ BcgShared sh;
  const int k = c.nrhs, tid = int(threadIdx.x);
  // Vector phases: thread t takes runs of V entries t, t + used, ... of the
  // CTA's chunks; used is a multiple of the runs per row, so its columns are
  // fixed.
  const int kv = k / V, used = CBS / kv * kv;
  const RV vr(tid % kv, k);
  const int c0 = vr.c0;
  const int64_t step = int64_t(used) * V;
  auto each = [&](auto&& body) {
    if (tid < used)
      for (int q = blockIdx.x; q < ch.count; q += gridDim.x) {
        const int64_t e1 = ch.end(q) * k;
#pragma unroll 2
        for (int64_t e = ch.begin(q) * k + int64_t(tid) * V; e < e1; e += step) body(e);
      }
  };
  unsigned long long epoch = 0;
  double acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.0;
  each([&](int64_t e) {
    double bv[V], z[V];
    ld_run<double>(vr, c.b + e, bv);
#pragma unroll
    for (int i = 0; i < V; ++i) {
      z[i] = 0.0;
      acc[i] += bv[i] * bv[i];
    }
    st_run<double>(vr, c.r + e, bv);
    st_run<double>(vr, c.p + e, bv);
    st_run<double>(vr, c.x + e, z);
  });
  // Consecutive sums publish into two arrays in turn: a CTA that runs ahead
  // never overwrites partials another still reads.
  auto parts = [&]() { return c.partials + (epoch & 1) * size_t(MAXK) * gridDim.x; };
  ++epoch;
  bool ok = column_sums<V>(acc, kv, used, c, parts(), epoch * gridDim.x, sh);
  int go = 0;
  if (tid < k) {
    const double rr = sh.tot[tid];
    sh.rr0[tid] = sh.rr[tid] = rr;
    sh.alpha[tid] = sh.beta[tid] = 0.0;
    sh.active[tid] = rr > 0.0 && isfinite(rr);
    sh.status[tid] = SPMV_SUCCESS;
    sh.its[tid] = 0;
    go = sh.active[tid];
  }
  go = __syncthreads_or(go) && ok && c.kmax > 0;
  for (int it = 1; go; ++it) {
    // A.  A thread's right-hand sides follow from its lane: tid % KL.
    double py[R::V];
#pragma unroll
    for (int i = 0; i < R::V; ++i) py[i] = 0.0;
    for (int q = blockIdx.x; q < ch.count; q += gridDim.x)
      each_rank(a, ch.begin(q), ch.end(q), [&](const PartArg& Q, int lo, int hi) {
        spmm_rows<double, CBS, KL, R>(
            Q, k, lo, hi, [&](const PartArg& P, int row, const R& run, const double(&s)[R::V]) {
              const int64_t o = int64_t(row) * k + run.c0;
              double pv[R::V];
              ld_run<double>(run, static_cast<const double*>(P.xown) + o, pv);
              st_run<double>(run, static_cast<double*>(P.y) + o, s);
#pragma unroll
              for (int i = 0; i < R::V; ++i) py[i] += pv[i] * s[i];
            });
      });
    ++epoch;
    if (!column_sums<R::V>(py, KL, CBS, c, parts(), epoch * gridDim.x, sh)) break;
    if (tid < k) {
      double alpha = 0.0;
      if (sh.active[tid]) {
        const double pap = sh.tot[tid];
        if (pap == 0.0 || !isfinite(pap)) {
          sh.status[tid] = SPMV_ERROR_BREAKDOWN;
          sh.active[tid] = 0;
        } else {
          alpha = sh.rr[tid] / pap;
        }
      }
      sh.alpha[tid] = alpha;
    }
    __syncthreads();
    // B.
    double al[V], be[V];
    bool act[V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      act[i] = sh.active[c0 + i];
      al[i] = sh.alpha[c0 + i];
      acc[i] = 0.0;
    }
    each([&](int64_t e) {
      double rv[V], yv[V];
      ld_run<double>(vr, c.r + e, rv);
      ld_run<double>(vr, c.y + e, yv);
#pragma unroll
      for (int i = 0; i < V; ++i)
        if (act[i]) {
          rv[i] = rv[i] - al[i] * yv[i];
          acc[i] += rv[i] * rv[i];
        }
      st_run<double>(vr, c.r + e, rv);
    });
    ++epoch;
    if (!column_sums<V>(acc, kv, used, c, parts(), epoch * gridDim.x, sh)) break;
    go = 0;
    // A column that stops in this iteration still takes C's x update.
    if (tid < k) {
      if (sh.active[tid]) {
        const double rr = sh.tot[tid];
        sh.its[tid] = it;
        sh.beta[tid] = rr / sh.rr[tid];
        sh.rr[tid] = rr;
        if (rr / sh.rr0[tid] < c.rtol2) sh.active[tid] = 0;
      } else {
        sh.beta[tid] = 0.0;
      }
      go = sh.active[tid] && it < c.kmax;
    }
    go = __syncthreads_or(go);
    // C.
#pragma unroll
    for (int i = 0; i < V; ++i) be[i] = sh.beta[c0 + i];
    each([&](int64_t e) {
      double xv[V], pv[V], rv[V];
      ld_run<double>(vr, c.x + e, xv);
      ld_run<double>(vr, c.p + e, pv);
      ld_run<double>(vr, c.r + e, rv);
#pragma unroll
      for (int i = 0; i < V; ++i)
        if (act[i]) {
          xv[i] = xv[i] + al[i] * pv[i];
          pv[i] = rv[i] + be[i] * pv[i];
        }
      st_run<double>(vr, c.x + e, xv);
      st_run<double>(vr, c.p + e, pv);
    });
    if (!go) break;
    ++epoch;
    __syncthreads();
    if (tid == 0) sh.ok = grid_arrive_wait(&c.st->bar, epoch * gridDim.x, &c.st->err, c.wait_ns);
    __syncthreads();
    if (!sh.ok) break;
  }
  if (blockIdx.x == 0 && tid < k) {
    c.st->rr0[tid] = sh.rr0[tid];
    c.st->rr[tid] = sh.rr[tid];
    c.st->status[tid] = sh.status[tid];
    c.st->its[tid] = sh.its[tid];
  }
}

// Lanes per row for k right-hand sides at v per lane.
int lanes_for(int k, int v) {
  int kl = 1;
  while (kl * v < k) kl <<= 1;
  return kl;
}

// Right-hand sides per lane: the widest run of at most 16 bytes that divides
// k and to which every vector is aligned; two loaded one by one (0) when k is
// odd or a vector is not aligned to two values.
int run_width(int k, size_t es, int P, const void* const* x, const void* const* y) {
  uintptr_t bits = 0;
  for (int r = 0; r < P; ++r) bits |= reinterpret_cast<uintptr_t>(x[r]) |
                                      reinterpret_cast<uintptr_t>(y[r]);
  if (k == 1) return 1;
  int v = int(16 / es);
  while (v > 1 && (k % v != 0 || bits % (v * es) != 0)) v /= 2;
  return v > 1 ? v : 0;
}

// Rows per chunk: at most `most`, so that the chunks are whole rounds of `grid` CTAs, of
// which `lost` may go to ranks that do not end with a whole chunk.
int64_t chunk_rows(int64_t total, int grid, int64_t most, int lost) {
  const int64_t rounds = std::max<int64_t>(1, (total + grid * most - 1) / (grid * most));
  const int64_t slots = std::max<int64_t>(1, grid * rounds - lost);
  return std::max<int64_t>(1, (total + slots - 1) / slots);
}
int64_t total_rows(spmv_matrix A) {
  int64_t total = 0;
  for (const DevPart& D : A->fwd.parts) total += D.nrows;
  return total;
}

// Block CG's chunks.
RowChunks row_chunks(spmv_matrix A, int grid, int64_t most) {
  RowChunks ch{};
  ch.total = total_rows(A);
  ch.rows = chunk_rows(ch.total, grid, most, 0);
  ch.count = int((ch.total + ch.rows - 1) / ch.rows);
  return ch;
}

template <typename T, class R>
const void* spmm_fn(int kl) {
  switch (kl) {
    case 1: return (const void*)spmm_kernel<T, 1, R>;
    case 2: return (const void*)spmm_kernel<T, 2, R>;
    case 4: return (const void*)spmm_kernel<T, 4, R>;
    case 8: return (const void*)spmm_kernel<T, 8, R>;
    case 16: if constexpr (R::V == 2) return (const void*)spmm_kernel<T, 16, R>;
  }
  fail(SPMV_ERROR_INTERNAL, "spmv: no block product for this width");
}

template <typename T>
const void* spmm_walk_fn(int kl) {
  switch (kl) {
    case 1: return (const void*)spmm_walk_kernel<T, 1>;
    case 2: return (const void*)spmm_walk_kernel<T, 2>;
    case 4: return (const void*)spmm_walk_kernel<T, 4>;
    case 8: return (const void*)spmm_walk_kernel<T, 8>;
    case 16: return (const void*)spmm_walk_kernel<T, 16>;
    case 32: return (const void*)spmm_walk_kernel<T, 32>;
  }
  fail(SPMV_ERROR_INTERNAL, "spmv: no block product for this width");
}

template <class R>
const void* bcg_fn(int kl) {
  switch (kl) {
    case 1: return (const void*)bcg_kernel<1, R>;
    case 2: return (const void*)bcg_kernel<2, R>;
    case 4: return (const void*)bcg_kernel<4, R>;
    case 8: return (const void*)bcg_kernel<8, R>;
    case 16: return (const void*)bcg_kernel<16, R>;
  }
  fail(SPMV_ERROR_INTERNAL, "spmv: no block solver for this width");
}

}  // namespace

// Whether a product with run width v (run_width) is spmm_walk_kernel's; us by it and by
// spmm_kernel:
//  * rows of several batches, single loads (odd k or unaligned vectors): twice the warps
//    are worth more than two right-hand sides per lane loaded one by one (FP64, 60^3 rows:
//    k = 7, 27-point 51 and 58, mesh 34 and 43; k = 31, 148 and 172, 91 and 102; rows of 7
//    entries, 96^3: k = 7, 70 and 66, k = 31, 255 and 219);
//  * rows of at most 4 entries, of which a batch of 8 repeats half (FP64, rows of 3: 600,000
//    k = 3 14.4 and 20.2, 2 M k = 3 58.8 and 64.2; FP32 600,000 k = 7 24.5 and 25.7, 2 M k
//    = 7 98.3 and 95.4, k = 17 358 and 304); in FP64 also the wide even k that leave lanes
//    over while X and Y stay in L2 (150,000 k = 24 24.6 and 29.0, 600,000 125 and 115);
//  * rows of at most 6 in FP64 while X and Y are well inside L2 (5-point 420^2 k = 7 12.3
//    and 14.4, 520^2 k = 3 10.3 and 12.3, 800^2 k = 5, 51 MB, 40.4 and 37.1);
//  * one right-hand side, a thread per row: rows of at most 6 entries (FP64 600,000 of 3
//    6.5 and 8.2, 1200^2 5-point 22.6 and 24.0, but 7-point 96^3 14.4 and 14.4, 40^3 5.2
//    and 4.1; FP32 2 M of 3 12.3 and 18.5), in FP32 of at most 8 where there are many
//    (7-point 88^3 8.8 and 9.3, 108^3 14.4 and 15.9, but 72^3 7.8 and 6.2).
static bool use_walk(const DevCsr& C, int64_t rows, int k, int v, size_t es, int l2_bytes) {
  if (C.max_row > LONG_ROW) return false;  // some row is for a whole CTA
  const bool f64 = es == 8;
  if (v == 0 && C.mean_row > SPMM_BATCH) return true;
  if (C.max_row > 4 * SPMM_BATCH) return false;
  const int64_t bytes = 2 * rows * k * int64_t(es);  // of X and Y
  if (k == 1) return C.mean_row <= (f64 || 32 * bytes <= l2_bytes ? 6.0 : 8.0);
  if (v != 0) return f64 && C.mean_row <= 4.0 && k > 8 && 2 * bytes <= l2_bytes;
  if (C.mean_row <= 4.0) return f64 || k < 16;
  return f64 && C.mean_row <= 6.0 && 4 * bytes <= l2_bytes;
}

// y[r] (nrows x k) = A[r] x[r] (ncols x k) for all ranks, device pointers.
void launch_spmm(spmv_matrix A, int k, const void* const* x, void* const* y,
                 cudaStream_t stream) {
  require(k >= 1 && k <= MAXK, "spmv: block products take 1..32 right-hand sides");
  require(A->dtype == SPMV_FLOAT64 || A->dtype == SPMV_FLOAT32,
          "spmv: only float64 and float32 products are implemented");
  const size_t es = dtype_size(A->dtype);
  const int v = run_width(k, es, A->comm->size, x, y);
  const bool f64 = A->dtype == SPMV_FLOAT64;
  if (use_walk(A->fwd, total_rows(A), k, v, es, A->comm->l2_bytes)) {
    const int kl = lanes_for(k, 1);
    SpmvArgs t;
    fill_spmv_args(t, A->fwd, A->fwd.cols.as<int32_t>(), es, x, y, nullptr, BBS / kl,
                   max_blocks_for(A->comm->num_sms, BBS));
    if (t.nblocks == 0) return;
    void* args[] = {&t, &k};
    SPMVB_CUDA(cudaLaunchKernel(f64 ? spmm_walk_fn<double>(kl) : spmm_walk_fn<float>(kl),
                                dim3(t.nblocks), dim3(BBS), args, 0, stream));
    return;
  }
  const int kl = lanes_for(k, v ? v : 2);
  const void* fn;
  if (k == 1)
    fn = f64 ? (const void*)spmm_kernel<double, 1, Run<1, false>>
             : (const void*)spmm_kernel<float, 1, Run<1, false>>;
  else if (f64)
    fn = v == 2 ? spmm_fn<double, Run<2, false>>(kl) : spmm_fn<double, Run<2, true>>(kl);
  else
    fn = v == 4   ? spmm_fn<float, Run<4, false>>(kl)
         : v == 2 ? spmm_fn<float, Run<2, false>>(kl)
                  : spmm_fn<float, Run<2, true>>(kl);
  // Chunks in flight are consecutive, so the X rows that rows further apart share (the
  // next plane of a grid) are read from DRAM once.
  int rows = int(chunk_rows(total_rows(A), std::max(1, A->comm->num_sms) * BCPS,
                            std::max(128, SPMM_CHUNK / k), A->comm->size - 1));
  SpmvArgs a;
  fill_spmv_args(a, A->fwd, A->fwd.cols.as<int32_t>(), es, x, y, nullptr, rows, INT32_MAX);
  if (a.nblocks == 0) return;
  void* args[] = {&a, &rows, &k};
  SPMVB_CUDA(cudaLaunchKernel(fn, dim3(a.nblocks), dim3(BBS), args, 0, stream));
}

void destroy_block_workspace(BlockWorkspace* w) { delete w; }

BlockWorkspace& block_workspace(spmv_matrix A) {
  if (!A->blk)
    A->blk = std::unique_ptr<BlockWorkspace, void (*)(BlockWorkspace*)>(new BlockWorkspace,
                                                                        destroy_block_workspace);
  return *A->blk;
}

void reserve_block(spmv_matrix A, BlockWorkspace& w, int k) {
  w.n = A->row_map->ranges.back();
  const size_t bytes = sizeof(double) * std::max<int64_t>(w.n * k, 1);
  for (DevBuf* v : w.vectors()) v->reserve(bytes);
  w.state.reserve(sizeof(BcgState));
  w.partials.reserve(sizeof(double) * 2 * MAXK * size_t(std::max(1, A->comm->num_sms)));
}

// At the end of a solve (also a failed one): vectors of up to BCG_KEEP bytes stay
// with the matrix for the next one, larger ones go back to the device.
struct BlockVectors {
  BlockWorkspace& w;
  ~BlockVectors() {
    size_t bytes = 0;
    for (DevBuf* v : w.vectors()) bytes += v->bytes;
    if (bytes > BCG_KEEP)
      for (DevBuf* v : w.vectors()) v->release();
  }
};

// Block CG in the fused-halo layout over the workspace's row-major n x k
// blocks: w.b to w.x.
void block_cg(spmv_matrix A, BlockWorkspace& w, int k, int max_its, double rtol,
              spmv_cg_info* info) {
  spmv_comm comm = A->comm;
  build_global_cols(A);
  const int P = comm->size;
  std::vector<const void*> xs(P), own(P);
  std::vector<void*> ys(P);
  for (int q = 0; q < P; ++q) {
    const int64_t off = A->row_map->ranges[q] * k;
    xs[q] = w.p.as<double>();
    own[q] = w.p.as<double>() + off;
    ys[q] = w.y.as<double>() + off;
  }
  SpmvArgs a;
  fill_spmv_args(a, A->fwd, A->fwd.cols_global.as<int32_t>(), sizeof(double), xs.data(), ys.data(),
                 own.data(), BBS, 1);
  BcgPtrs c{};
  c.b = w.b.as<double>();
  c.x = w.x.as<double>();
  c.r = w.r.as<double>();
  c.p = w.p.as<double>();
  c.y = w.y.as<double>();
  c.partials = w.partials.as<double>();
  c.st = w.state.as<BcgState>();
  c.nrhs = k;
  c.kmax = max_its;
  c.rtol2 = rtol * rtol;
  c.wait_ns = fused_wait_ns();
  cudaStream_t s = comm->stream;
  const int kl = lanes_for(k, 2);
  const void* fn = k == 1       ? (const void*)bcg_kernel<1, Run<1, false>>
                   : k % 2 == 0 ? bcg_fn<Run<2, false>>(kl)
                                : bcg_fn<Run<2, true>>(kl);
  // Every CTA resident; a device that cannot hold the grid at once (a context
  // with fewer SMs) gets a smaller one.
  int grid = std::max(1, comm->num_sms);
  for (;;) {
    SPMVB_CUDA(cudaMemsetAsync(c.st, 0, sizeof(BcgState), s));
    RowChunks ch = row_chunks(A, grid, std::max(128, BCG_CHUNK / k));
    void* args[] = {&a, &c, &ch};
    const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(CBS), args, 0, s);
    if (e != cudaErrorCooperativeLaunchTooLarge || grid == 1) {
      SPMVB_CUDA(e);
      break;
    }
    (void)cudaGetLastError();
    grid = (grid + 1) / 2;
  }
  BcgState host{};
  SPMVB_CUDA(cudaMemcpyAsync(&host, c.st, sizeof(BcgState), cudaMemcpyDeviceToHost, s));
  SPMVB_CUDA(cudaStreamSynchronize(s));
  if (host.err) fail(SPMV_ERROR_CUDA, "spmv::cg - a bounded wait of the block solve timed out");
  for (int l = 0; l < k; ++l) {
    info[l].iterations = host.its[l];
    info[l].status = host.status[l];
    info[l].rnorm0 = host.rr0[l];
    info[l].rnorm = host.rr[l];
  }
}

}  // namespace spmvb

using namespace spmvb;

extern "C" {

int spmv_matrix_mult_block(spmv_matrix A, int nrhs, spmv_memory memory,
                           const void* const* x, void* const* y) {
  return guard([&] {
    require(A != nullptr, "spmv: Matrix is NULL");
    require(x != nullptr && y != nullptr, "spmv: vector array is NULL");
    require(nrhs >= 1 && nrhs <= MAXK, "spmv: block products take 1..32 right-hand sides");
    spmv_comm comm = A->comm;
    comm->require_device();
    DeviceGuard dg(comm->device);
    cudaStream_t s = comm->stream;
    if (memory == SPMV_MEMORY_DEVICE) {
      launch_spmm(A, nrhs, x, y, s);
      return;
    }
    require(memory == SPMV_MEMORY_HOST, "spmv: unknown memory kind");
    const int P = comm->size;
    const size_t es = dtype_size(A->dtype);
    std::vector<int64_t> xo(P), yo(P);
    int64_t xt = 0, yt = 0;
    for (int r = 0; r < P; ++r) {
      xo[r] = xt;
      yo[r] = yt;
      xt += (int64_t(A->ncols[r]) * nrhs * es + 255) / 256 * 256;
      yt += (int64_t(A->nrows[r]) * nrhs * es + 255) / 256 * 256;
    }
    comm->stage_in.reserve(std::max<int64_t>(xt, 256));
    comm->stage_out.reserve(std::max<int64_t>(yt, 256));
    std::vector<const void*> dx(P);
    std::vector<void*> dy(P);
    for (int r = 0; r < P; ++r) {
      dx[r] = comm->stage_in.as<char>() + xo[r];
      dy[r] = comm->stage_out.as<char>() + yo[r];
      const size_t bytes = size_t(A->ncols[r]) * nrhs * es;
      if (bytes)
        SPMVB_CUDA(cudaMemcpyAsync(const_cast<void*>(dx[r]), x[r], bytes,
                                   cudaMemcpyHostToDevice, s));
    }
    launch_spmm(A, nrhs, dx.data(), dy.data(), s);
    for (int r = 0; r < P; ++r) {
      const size_t bytes = size_t(A->nrows[r]) * nrhs * es;
      if (bytes) SPMVB_CUDA(cudaMemcpyAsync(y[r], dy[r], bytes, cudaMemcpyDeviceToHost, s));
    }
    SPMVB_CUDA(cudaStreamSynchronize(s));
  });
}

int spmv_cg_block(spmv_matrix A, int nrhs, spmv_memory memory, const double* const* b,
                  double* const* x, int max_its, double rtol, spmv_cg_info* info) {
  return guard([&] {
    require(nrhs >= 1 && nrhs <= MAXK, "spmv: block CG takes 1..32 right-hand sides");
    check_solve_args(A, memory, b, nullptr, x);
    spmv_comm comm = A->comm;
    DeviceGuard dg(comm->device);
    cudaStream_t s = comm->stream;
    spmv_l2gmap rm = A->row_map, cm = A->col_map;
    const int P = comm->size;
    BlockWorkspace& w = block_workspace(A);
    const BlockVectors vectors{w};
    reserve_block(A, w, nrhs);
    const cudaMemcpyKind in = memory == SPMV_MEMORY_HOST ? cudaMemcpyHostToDevice
                                                         : cudaMemcpyDeviceToDevice;
    const cudaMemcpyKind outk = memory == SPMV_MEMORY_HOST ? cudaMemcpyDeviceToHost
                                                           : cudaMemcpyDeviceToDevice;
    for (int r = 0; r < P; ++r) {
      const int64_t M = rm->rank[r].local_size;
      if (M == 0) continue;
      require(b[r] != nullptr, "spmv::cg - Error: b is NULL");
      SPMVB_CUDA(cudaMemcpyAsync(w.b.as<double>() + rm->ranges[r] * nrhs, b[r],
                                 sizeof(double) * M * nrhs, in, s));
    }
    std::vector<spmv_cg_info> local(nrhs);
    block_cg(A, w, nrhs, max_its, rtol, local.data());
    for (int r = 0; r < P; ++r) {
      const int64_t M = rm->rank[r].local_size;
      const int64_t G = int64_t(cm->rank[r].ghosts.size());
      if (M + G == 0) continue;
      require(x[r] != nullptr, "spmv::cg - Error: x is NULL");
      if (M > 0)
        SPMVB_CUDA(cudaMemcpyAsync(x[r], w.x.as<double>() + rm->ranges[r] * nrhs,
                                   sizeof(double) * M * nrhs, outk, s));
      if (G > 0) {
        if (memory == SPMV_MEMORY_HOST)
          std::fill(x[r] + M * nrhs, x[r] + (M + G) * nrhs, 0.0);
        else
          SPMVB_CUDA(cudaMemsetAsync(x[r] + M * nrhs, 0, sizeof(double) * G * nrhs, s));
      }
    }
    SPMVB_CUDA(cudaStreamSynchronize(s));
    if (info) std::copy(local.begin(), local.end(), info);
    for (int l = 0; l < nrhs; ++l)
      if (local[l].status == SPMV_ERROR_BREAKDOWN)
        fail(SPMV_ERROR_BREAKDOWN, "spmv::cg - Error: breakdown in right-hand side " +
                                       std::to_string(l));
  });
}

}  // extern "C"
