// Merge-path CSR product: load-balanced for skewed row lengths.
//
// The product is the merge of two lists, the row ends rowptr[1..m] and the
// entry indices 0..nnz-1 (m + nnz items; Merrill & Garland, "Merge-based
// parallel sparse matrix-vector multiplication", SC'16).  Consuming an entry
// adds v[j] * x[c[j]] to the current row's sum; consuming a row end emits the
// row.  Every CTA takes an equal tile of TILE = BS * IPT consecutive items,
// whatever the row lengths, so one long row is spread over many CTAs.
//
// Per CTA: a search on the diagonal gives the tile's first and last (row, entry)
// coordinates; the tile's products and row ends are staged in shared memory with
// coalesced loads; then each row's part in the tile is summed: up to SHORT
// entries by one thread in storage order, up to MID by a warp, more by the
// CTA, so neither many short rows nor one long one leaves the CTA waiting.
// Rows that end in the tile are stored (their part of it), the sum of the row
// the tile ends in goes to a per-CTA carry, and merge_fixup adds each run of
// carries that belong to one row, in CTA order, to that row.  Every order is
// fixed, so results are reproducible.
//
// What bounded it: two threads' binary searches before any load (18 dependent
// loads), and a merge walk of 8 items per thread through shared memory, each
// item two reads in diverging branches.  300,007 power-law rows (3.8 M
// entries, the longest 37,500) in FP64: 57 -> 35 us per product with the search
// by a warp, loads in one batch per thread and the sums by row.
#include <algorithm>
#include <mutex>
#include <string>
#include <vector>

#include "internal.h"
#include "kernels.cuh"

namespace spmvb {

namespace {

constexpr int MBS = 256;  // threads per CTA
constexpr int IPT = 8;    // merge items per thread
constexpr int TILE = MBS * IPT;
// Entries of a tile that one thread sums, and one warp.  A thread per row is the
// fastest where the rows' lengths are odd multiples of few banks (4 M entries, us per
// product: rows of 17, 18.5 with SHORT = 32 and 39.0 with 16; of 33, 28.7 and with 64
// 18.5; but of 32, 31.2 and with 16 28.7, of 64, 22.6 and with 64 32.7: the lanes of
// equal rows then share banks).  MID = 128: rows of 200 31.5 against 18.5; MID = 512: of
// 300 17.8 against 26.6, of 600 20.8 against 22.4; 300,007 power-law rows 34.6, between
// 33.8 and 36.5 with any of these.
constexpr int SHORT = 32;
constexpr int MID = 256;

// Smallest row count i in [lo, hi] (rows consumed) of the split point on
// diagonal d: the first i with rowend(i) > d - i - 1, rowend(i) = rowptr[i + 1].
// A whole warp searches: each step probes 32 places between lo and hi, so over
// 300,000 rows it is 4 dependent loads instead of 18.
__device__ __forceinline__ int merge_search_warp(int d, int lo, int hi,
                                                 const int32_t* __restrict__ rowptr) {
  const int lane = int(threadIdx.x) & 31;
  while (lo < hi) {
    // Probe lo + (lane + 1) * step - 1; the condition holds for a prefix.
    const int step = (hi - lo + 31) >> 5;
    const int at = lo + (lane + 1) * step - 1;
    const bool past = at < hi && __ldg(rowptr + at + 1) <= d - at - 1;
    const int n = __popc(__ballot_sync(0xffffffffu, past));
    lo += n * step;               // the last probe of the prefix is consumed
    hi = min(hi, lo + step - 1);  // and the next one is not
  }
  return lo;
}

template <typename T>
__global__ void __launch_bounds__(MBS)
    merge_kernel(const __grid_constant__ SpmvArgs a, int* __restrict__ carry_row,
                 T* __restrict__ carry_val) {
  __shared__ int s_rp[TILE + 2];
  __shared__ T s_prod[TILE];
  __shared__ T s_red[MBS / 32];
  __shared__ T s_carry;
  __shared__ int s_bounds[4], s_nmid, s_nbig;
  __shared__ int s_mid[TILE / (SHORT + 1) + 1], s_big[TILE / (MID + 1) + 1];

  const int p = find_part(a, blockIdx.x);
  const PartArg& P = a.part[p];
  const int m = P.nrows;
  const int32_t* __restrict__ rowptr = P.rowptr;
  const int nnz = rowptr[m];
  const long total = long(m) + nnz;
  const int tile = int(blockIdx.x) - P.block_begin;
  const long d0l = long(tile) * TILE;
  const int d0 = int(d0l);
  const int d1 = int(min(total, d0l + TILE));
  const int lane = int(threadIdx.x) & 31, warp = int(threadIdx.x) >> 5;

  if (threadIdx.x == 0) {
    s_carry = T(0);
    s_nmid = s_nbig = 0;
  }
  if (warp < 2) {
    const int d = warp == 0 ? d0 : d1;
    const int i = merge_search_warp(d, max(0, d - nnz), min(d, m), rowptr);
    if (lane == 0) {
      s_bounds[2 * warp] = i;
      s_bounds[2 * warp + 1] = d - i;
    }
  }
  __syncthreads();
  const int i0 = s_bounds[0], j0 = s_bounds[1];
  const int i1 = s_bounds[2], j1 = s_bounds[3];

  // Row pointers i0 .. min(i1 + 1, m) and products j0 .. j1-1.  The
  // products in one batch of IPT loads per thread (past the tile's last entry
  // a thread repeats it).
  const int nr = min(i1 + 1, m) - i0 + 1;
  for (int k = threadIdx.x; k < nr; k += MBS) s_rp[k] = __ldg(rowptr + i0 + k);
  const T* __restrict__ vals = static_cast<const T*>(P.vals);
  const T* __restrict__ x = static_cast<const T*>(P.x);
  const int nj = j1 - j0;
  if (nj > 0) {
    int c[IPT];
    T v[IPT];
#pragma unroll
    for (int q = 0; q < IPT; ++q) {
      const int j = j0 + min(int(threadIdx.x) + q * MBS, nj - 1);
      c[q] = ld_stream(P.cols + j);
      v[q] = ld_stream(vals + j);
    }
    T xv[IPT];
#pragma unroll
    for (int q = 0; q < IPT; ++q) xv[q] = ld_gather(x + c[q]);
#pragma unroll
    for (int q = 0; q < IPT; ++q)
      if (int(threadIdx.x) + q * MBS < nj) s_prod[threadIdx.x + q * MBS] = v[q] * xv[q];
  }
  pdl_launch_dependents();  // merge_fixup may be scheduled; it waits for this kernel's end
  __syncthreads();

  // Row q of the tile (row i0 + q): its products [b, e) in s_prod; the last one
  // (row i1) does not end here.
  const int nrows = i1 - i0 + (i1 < m ? 1 : 0);
  auto range = [&](int q, int& b, int& e) {
    b = max(s_rp[q], j0) - j0;
    e = min(s_rp[q + 1], j1) - j0;
  };
  T* __restrict__ y = static_cast<T*>(P.y);
  auto store = [&](int q, T sum) {
    if (i0 + q < i1)
      y[i0 + q] = sum;
    else
      s_carry = sum;
  };
  for (int q = int(threadIdx.x); q < nrows; q += MBS) {
    int b, e;
    range(q, b, e);
    if (e - b > MID) {
      s_big[atomicAdd(&s_nbig, 1)] = q;
    } else if (e - b > SHORT) {
      s_mid[atomicAdd(&s_nmid, 1)] = q;
    } else {
      T sum = T(0);
      for (int k = b; k < e; ++k) sum += s_prod[k];
      store(q, sum);
    }
  }
  __syncthreads();
  for (int l = warp; l < s_nmid; l += MBS / 32) {
    int b, e;
    range(s_mid[l], b, e);
    T sum = T(0);
    for (int k = b + lane; k < e; k += 32) sum += s_prod[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) store(s_mid[l], sum);
  }
  for (int l = 0; l < s_nbig; ++l) {
    int b, e;
    range(s_big[l], b, e);
    T sum = T(0);
    for (int k = b + int(threadIdx.x); k < e; k += MBS) sum += s_prod[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) s_red[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
      sum = s_red[0];
#pragma unroll
      for (int w = 1; w < MBS / 32; ++w) sum += s_red[w];
      store(s_big[l], sum);
    }
    __syncthreads();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    carry_row[blockIdx.x] = i1 < m ? i1 : -1;
    carry_val[blockIdx.x] = s_carry;
  }
}

// Adds the carries of CTAs that ended inside a row to that row, one thread
// per run of equal (rank, row) carries, summed in CTA order.
template <typename T>
__global__ void merge_fixup(const __grid_constant__ SpmvArgs a,
                            const int* __restrict__ carry_row,
                            const T* __restrict__ carry_val, int nblocks) {
  pdl_wait();  // launched programmatically behind merge_kernel
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nblocks) return;
  const int r = carry_row[c];
  if (r < 0) return;
  const int p = find_part(a, c);
  if (c > a.part[p].block_begin && carry_row[c - 1] == r) return;  // not a run start
  const int end = a.part[p].block_begin + a.part[p].nblocks;
  T acc = T(0);
  int e = c;
  while (e < end && carry_row[e] == r) acc += carry_val[e++];
  T* y = static_cast<T*>(a.part[p].y);
  y[r] = y[r] + acc;
}

}  // namespace

// merge_kernel and merge_fixup over a table of `blocks` tiles.
template <typename T>
void launch_tiles(const SpmvArgs& a, int blocks, int* crow, T* cval, cudaStream_t s) {
  merge_kernel<T><<<blocks, MBS, 0, s>>>(a, crow, cval);
  SPMVB_CUDA(cudaGetLastError());
  const int* cr = crow;
  const T* cv = cval;
  void* args[] = {const_cast<SpmvArgs*>(&a), &cr, &cv, &blocks};
  launch_pdl((const void*)merge_fixup<T>, dim3((blocks + 255) / 256), dim3(256), 0, s, args);
}

void launch_merge(const SpmvLaunch& L, cudaStream_t stream, DevBuf& carry) {
  const DevCsr& C = *L.csr;
  const size_t es = dtype_size(L.dtype);
  SpmvArgs a;
  a.nparts = int(C.parts.size());
  int blocks = 0;
  for (int p = 0; p < a.nparts; ++p) {
    const DevPart& D = C.parts[p];
    PartArg& P = a.part[p];
    P.rowptr = C.rowptr.as<int32_t>() + D.rp_off;
    P.cols = L.cols + D.nz_off;
    P.vals = static_cast<const char*>(C.vals.ptr) + D.nz_off * es;
    P.x = L.x[p];
    P.y = L.y[p];
    P.xown = nullptr;
    P.nrows = D.nrows;
    P.block_begin = blocks;
    const int64_t items = int64_t(D.nrows) + D.nnz;
    require(items < (int64_t(1) << 31) - TILE, "spmv: rank too large for merge-path");
    const int64_t nb = (items + TILE - 1) / TILE;
    P.nblocks = int32_t(nb);
    P.ntiles = int32_t(nb);
    require(blocks + nb < (int64_t(1) << 31), "spmv: too many tiles");
    blocks += int(nb);
  }
  a.nblocks = blocks;
  if (blocks == 0) return;
  carry.reserve(size_t(blocks) * (sizeof(int) + 8) + 256);
  int* crow = carry.as<int>();
  void* cval = carry.as<char>() + ((size_t(blocks) * sizeof(int) + 255) / 256) * 256;
  if (L.dtype == SPMV_FLOAT64)
    launch_tiles(a, blocks, crow, static_cast<double*>(cval), stream);
  else
    launch_tiles(a, blocks, crow, static_cast<float*>(cval), stream);
}

// ---------------------------------------------------------------------------
// Allocation-free product: spmv_matrix_mult_noalloc.
//
// The merge-path product above keeps its per-CTA carries in a buffer that
// spmv_matrix_mult allocates (and grows) on demand.  This variant runs the
// same two kernels with the carries in a fixed file-scope device array, so a
// call allocates no device memory.  The array holds NOALLOC_MAX_TILES tiles of
// TILE (= 2048) merge items, i.e. rows + nonzeros of all ranks together up to
// 16384 * 2048 = 33,554,432; it is 192 KiB and stays resident on every
// device that loads this library until the process exits.
// ---------------------------------------------------------------------------
constexpr int NOALLOC_MAX_TILES = 16384;
constexpr size_t NOALLOC_VAL_OFFSET = size_t(NOALLOC_MAX_TILES) * sizeof(int);
static __device__ __align__(256) unsigned char
    g_noalloc_carry[NOALLOC_VAL_OFFSET + size_t(NOALLOC_MAX_TILES) * sizeof(double)];

namespace {

// Device address of g_noalloc_carry, looked up once per device (with that
// device current).  Host code must not use the symbol's name as an address:
// on the host it names a shadow object, not device memory.  The cached
// address belongs to the device's primary context as it was at the first
// call; a cudaDeviceReset ends that context (and every handle of this
// library made in it), so the cache is not meant to outlive one.
void* noalloc_scratch(int device) {
  static std::mutex mu;
  static std::vector<void*> addr;
  std::lock_guard<std::mutex> lock(mu);
  if (int(addr.size()) <= device) addr.resize(device + 1, nullptr);
  if (!addr[device]) {
    void* p = nullptr;
    SPMVB_CUDA(cudaGetSymbolAddress(&p, g_noalloc_carry));
    addr[device] = p;
  }
  return addr[device];
}

}  // namespace

}  // namespace spmvb

extern "C" int spmv_matrix_mult_noalloc(spmv_matrix A, const void* const* x,
                                        void* const* y) {
  using namespace spmvb;
  return guard([&] {
    require(A != nullptr, "spmv: Matrix is NULL");
    require(x != nullptr && y != nullptr, "spmv: vector array is NULL");
    require(A->dtype == SPMV_FLOAT64 || A->dtype == SPMV_FLOAT32,
            "spmv: only float64 and float32 products are implemented");
    const DevCsr& C = A->fwd;
    const size_t es = dtype_size(A->dtype);
    SpmvArgs a;
    a.nparts = int(C.parts.size());
    int64_t blocks = 0;
    for (int p = 0; p < a.nparts; ++p) {
      const DevPart& D = C.parts[p];
      if (D.ncols > 0) require(x[p] != nullptr, "spmv: x vector is NULL");
      if (D.nrows > 0) require(y[p] != nullptr, "spmv: y vector is NULL");
      const int64_t nb = (int64_t(D.nrows) + D.nnz + TILE - 1) / TILE;
      PartArg& P = a.part[p];
      P.rowptr = C.rowptr.as<int32_t>() + D.rp_off;
      P.cols = C.cols.as<int32_t>() + D.nz_off;
      P.vals = static_cast<const char*>(C.vals.ptr) + D.nz_off * es;
      P.x = x[p];
      P.y = y[p];
      P.xown = nullptr;
      P.nrows = D.nrows;
      P.block_begin = int32_t(std::min<int64_t>(blocks, NOALLOC_MAX_TILES));
      P.nblocks = int32_t(std::min<int64_t>(nb, NOALLOC_MAX_TILES));
      P.ntiles = P.nblocks;
      blocks += nb;
    }
    if (blocks > NOALLOC_MAX_TILES)
      fail(SPMV_ERROR_INVALID_ARGUMENT,
           "spmv_matrix_mult_noalloc: rows + nonzeros over all ranks (" +
               std::to_string(blocks) + " tiles of 2048) exceed the maximum of " +
               std::to_string(NOALLOC_MAX_TILES) + " tiles (33554432 items)");
    a.nblocks = int(blocks);
    A->comm->require_device();
    DeviceGuard dg(A->comm->device);
    if (blocks == 0) return;
    unsigned char* base = static_cast<unsigned char*>(noalloc_scratch(A->comm->device));
    int* crow = reinterpret_cast<int*>(base);
    cudaStream_t s = A->comm->stream;
    // Every CTA writes its carry slot before the fix-up reads it, so the
    // array needs no clearing between calls.
    if (A->dtype == SPMV_FLOAT64)
      launch_tiles(a, int(blocks), crow, reinterpret_cast<double*>(base + NOALLOC_VAL_OFFSET), s);
    else
      launch_tiles(a, int(blocks), crow, reinterpret_cast<float*>(base + NOALLOC_VAL_OFFSET), s);
  });
}
