// SELL-32 traversal with a private ring of shared-memory slots per warp.
//
// A warp takes whole items of S consecutive slices of a rank (one lane per row
// of each) and streams its own entries: a copy is a whole item (S = 2: two
// slices of at most U columns, adjacent in the SELL layout) or up to U columns
// of a slice (S = 1, so a wide slice is several copies), values then indices,
// into a slot by two bulk copies that complete on the slot's mbarrier.  A slot
// is refilled as soon as the warp has read it into registers, before the
// gathers of its entries have come back, so all the slots stay in flight; no
// other warp takes part, so there is nothing to deal out and no tile whose last
// slice the others wait for.  Entries are summed in storage order, so results
// are bitwise those of every SELL-32 product.
//
// Item table (host-built, S = 1 or 2): {first entry / 32, global row of the
// first lane, slices, 0} with slices = columns | rows << 24 (S = 1) or
// columns 0 | columns 1 << 8 | rows 0 << 16 | rows 1 << 24 (S = 2; an odd last
// slice leaves the second empty), all ranks in order; the CTA's part of it is
// in shared memory.
//
// Waits are bounded like the staged pipeline's (mbar_wait_bounded).
#pragma once

#include "sell_staged.cuh"

namespace spmvb {

constexpr int RING_MAX_COLS = (1 << 24) - 1;

// U columns per slice and S slices per slot, D slots per warp.
template <typename T, typename CI, int U, int D, int S>
struct RingShape {
  static constexpr int VB = S * U * 32 * int(sizeof(T)), IB = S * U * 32 * int(sizeof(CI));
  static constexpr int SLOT = VB + IB;
  static constexpr int BYTES = D * SLOT;  // one warp's slots
};

// What a warp's ring needs besides its state; kept out of registers where the
// caller can (kernel parameters, shared memory).
template <typename T, typename CI>
struct RingView {
  const T* vals;
  const CI* idx;
  const int4* items;    // shared memory: the CTA's items
  int count, stride;    // items of the CTA; the warp takes warp, warp + stride, ...
  unsigned char* base;  // the warp's slots
  uint64_t* bar;        // and their barriers
  const uint64_t* policy;  // the copies' L2 policy (shared memory)
};

// State of a warp's ring (registers).
struct RingState {
  int j, k;      // next copy: item, first column (S = 1)
  int fill, rd;  // next slot to fill, next slot to read
  uint32_t phase;
};

// One lane per warp (a barrier of the CTA follows before ring_prime).
template <int D>
__device__ __forceinline__ void ring_init(uint64_t* bar) {
#pragma unroll
  for (int s = 0; s < D; ++s) mbar_init(bar + s, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Whole warp.  The next copy of the warp's passes (the last of a pass is
// followed by the first of the next) into the next slot.
template <typename T, typename CI, int U, int D, int S>
__device__ __forceinline__ void ring_issue(const RingView<T, CI>& v, RingState& r) {
  using Sh = RingShape<T, CI, U, D, S>;
  const int4 d = v.items[r.j];
  const int w = S == 2 ? (d.z & 255) + ((d.z >> 8) & 255) : d.z & RING_MAX_COLS;
  if ((threadIdx.x & 31) == 0) {
    const uint32_t n = uint32_t(S == 2 ? w : min(U, w - r.k)) * 32u;
    const int64_t e = (int64_t(d.x) + (S == 2 ? 0 : r.k)) * 32;
    unsigned char* s = v.base + r.fill * Sh::SLOT;
    uint64_t* bar = v.bar + r.fill;
    mbar_arrive_expect_tx(bar, n * uint32_t(sizeof(T) + sizeof(CI)));
    if (n > 0) {
      const uint64_t policy = *v.policy;
      bulk_g2s(s, v.vals + e, n * uint32_t(sizeof(T)), bar, policy);
      bulk_g2s(s + Sh::VB, v.idx + e, n * uint32_t(sizeof(CI)), bar, policy);
    }
  }
  r.fill = r.fill + 1 == D ? 0 : r.fill + 1;
  if (S == 1) r.k += U;
  if (S == 2 || r.k >= w) {
    r.k = 0;
    r.j += v.stride;
    if (r.j >= v.count) r.j = int(threadIdx.x) >> 5;
  }
}

template <typename T, typename CI, int U, int D, int S>
__device__ __forceinline__ void ring_prime(const RingView<T, CI>& v, RingState& r) {
  r = RingState{int(threadIdx.x) >> 5, 0, 0, 0, 0u};
  if (r.j >= v.count) return;
#pragma unroll
  for (int s = 0; s < D; ++s) ring_issue<T, CI, U, D, S>(v, r);
}

// Before the CTA exits: waits (bounded) for the warp's copies in flight.
template <typename T, typename CI, int D>
__device__ __forceinline__ void ring_drain(const RingView<T, CI>& v, const RingState& r) {
  if (int(threadIdx.x) >> 5 >= v.count) return;
  for (int s = 0; s < D; ++s) mbar_wait_bounded(v.bar + s, (r.phase >> s) & 1u);
}

// The lane's rows of an item: global row and whether it exists.
template <int S>
struct RingRows {
  int g[S];
  bool valid[S];
  RingRows() = default;
  __device__ __forceinline__ explicit RingRows(const int4& h) {
    const int lane = int(threadIdx.x) & 31;
    if constexpr (S == 1) {
      g[0] = h.y + lane;
      valid[0] = lane < (h.z >> 24);
    } else {
      const int n0 = (h.z >> 16) & 255;
      g[0] = h.y + lane;
      g[1] = h.y + n0 + lane;
      valid[0] = lane < n0;
      valid[1] = lane < int(unsigned(h.z) >> 24);
    }
  }
};

// The landed slot: reads W columns per slice (W == U: `all`, no column masks;
// a padding entry then gathers entry 0, whose value is not used), hands the
// slot back and adds the products in storage order.  LATE: the values are read
// when they are used and the slot handed back after that (2 S U registers
// fewer).
template <typename T, typename CI, int U, int D, int S, bool LATE, bool ALL, class G>
__device__ __forceinline__ void ring_slot(const RingView<T, CI>& v, RingState& r,
                                          const unsigned char* slot, const int (&cols)[S],
                                          const int (&g)[S], const G& gx, T (&sum)[S]) {
  const int lane = int(threadIdx.x) & 31;
  const T* sv = reinterpret_cast<const T*>(slot) + lane;
  const CI* sc =
      reinterpret_cast<const CI*>(slot + RingShape<T, CI, U, D, S>::VB) + lane;
  T vv[LATE ? 1 : S][U], xv[S][U];
  bool ok[S][U];
#pragma unroll
  for (int q = 0; q < S; ++q)
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int at = (ALL ? q * U + u : (q == 0 ? u : cols[0] + u)) * 32;
      const bool in = ALL || u < cols[q];
      const int ci = in ? int(sc[at]) : (sizeof(CI) == 2 ? -32768 : -1);
      ok[q][u] = sizeof(CI) == 2 ? ci != -32768 : ci >= 0;
      const int c = sizeof(CI) == 2 ? g[q] + ci : ci;
      if (ALL)
        xv[q][u] = gx(ok[q][u] ? c : 0);
      else
        xv[q][u] = ok[q][u] ? gx(c) : T(0);
    }
  if constexpr (!LATE) {
#pragma unroll
    for (int q = 0; q < S; ++q)
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int at = (ALL ? q * U + u : (q == 0 ? u : cols[0] + u)) * 32;
        if (ALL)
          vv[q][u] = sv[at];
        else
          vv[q][u] = ok[q][u] ? sv[at] : T(0);
      }
    __syncwarp();  // the slot has been read by every lane
    ring_issue<T, CI, U, D, S>(v, r);
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int q = 0; q < S; ++q)
      if (ok[q][u]) {
        const int at = (ALL ? q * U + u : (q == 0 ? u : cols[0] + u)) * 32;
        if constexpr (LATE)
          sum[q] += sv[at] * xv[q][u];
        else
          sum[q] += vv[q][u] * xv[q][u];
      }
  if constexpr (LATE) {
    __syncwarp();
    ring_issue<T, CI, U, D, S>(v, r);
  }
}

// One pass over the warp's items: f(i, rows, sums) for its item i; gx(c): the
// gathered vector at column c (the column of an entry that exists, or 0).  CI int16: columns are offsets from the row,
// -32768 = padding; int32: columns, -1 = padding.  Returns false when a wait
// ran out.
template <typename T, typename CI, int U, int D, int S, bool LATE, class G, class F>
__device__ __forceinline__ bool ring_pass(const RingView<T, CI>& v, RingState& r, const G& gx,
                                          F&& f) {
  using Sh = RingShape<T, CI, U, D, S>;
  int i = 0;
  for (int j = int(threadIdx.x) >> 5; j < v.count; j += v.stride, ++i) {
    const int4 h = v.items[j];
    const RingRows<S> rows(h);
    T sum[S];
    int cols[S];
#pragma unroll
    for (int q = 0; q < S; ++q) {
      sum[q] = T(0);
      cols[q] = S == 1 ? h.z & RING_MAX_COLS : (h.z >> (8 * q)) & 255;
    }
    do {
      if (!mbar_wait_bounded(v.bar + r.rd, (r.phase >> r.rd) & 1u)) return false;
      const unsigned char* slot = v.base + r.rd * Sh::SLOT;
      r.phase ^= 1u << r.rd;
      r.rd = r.rd + 1 == D ? 0 : r.rd + 1;
      if (S == 1 ? cols[0] >= U : (h.z & 0xffff) == (U | U << 8))
        ring_slot<T, CI, U, D, S, LATE, true>(v, r, slot, cols, rows.g, gx, sum);
      else
        ring_slot<T, CI, U, D, S, LATE, false>(v, r, slot, cols, rows.g, gx, sum);
      cols[0] -= U;
    } while (S == 1 && cols[0] > 0);
    f(i, rows, sum);
  }
  return true;
}

// ---------------------------------------------------------------------------
// Tensor memory as storage for a warp's own vector entries: 32-bit columns of
// the warp's 32 lanes (warp w of the CTA owns lanes 32 (w % 4) ..), read and
// written by that warp only.
// ---------------------------------------------------------------------------
// One warp of the CTA, converged; the address is written to *slot (shared).
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_addr(slot)),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// 64-bit values in two columns.
struct Tmem64 {
  uint32_t lo, hi;
  __device__ __forceinline__ double get() const { return __hiloint2double(int(hi), int(lo)); }
};
__device__ __forceinline__ void tmem_ld(uint32_t addr, Tmem64& a) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];"
               : "=r"(a.lo), "=r"(a.hi)
               : "r"(addr));
}
__device__ __forceinline__ void tmem_st(uint32_t addr, double v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(addr),
               "r"(__double2loint(v)), "r"(__double2hiint(v))
               : "memory");
}
// 32-bit values in one column.
struct Tmem32 {
  uint32_t v;
  __device__ __forceinline__ float get() const { return __uint_as_float(v); }
};
__device__ __forceinline__ void tmem_ld(uint32_t addr, Tmem32& a) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(a.v) : "r"(addr));
}
__device__ __forceinline__ void tmem_st(uint32_t addr, float v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(addr),
               "r"(__float_as_uint(v))
               : "memory");
}
// A load's registers are valid after the wait.  tmem_wait_ld takes every value that
// is in flight and gives each of them back from behind the wait, so that nothing
// computed from one can be moved ahead of it.  The loads are unconditional, so that
// no copy of a register is made between a load and its wait.
__device__ __forceinline__ void tmem_landed(Tmem64& a) {
  asm volatile("" : "+r"(a.lo), "+r"(a.hi));
}
__device__ __forceinline__ void tmem_landed(Tmem32& a) { asm volatile("" : "+r"(a.v)); }
template <class R, int N>
__device__ __forceinline__ void tmem_landed(R (&a)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) tmem_landed(a[i]);
}
template <class... R>
__device__ __forceinline__ void tmem_wait_ld(R&... loaded) {
  static_assert(sizeof...(R) > 0, "the values that the wait is for");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  (tmem_landed(loaded), ...);
}

}  // namespace spmvb
