// nlgb_sell.cu -- row-sorted sliced matrix layout and its SpMV (FP64, two
// threads per row: the LSCM normal equations).
//
// Replaces, for large systems, the CRS walk of nlMultMatrixVector inside the
// solvers (src/lib/OGF/scene_graph/NL/matrix.cpp:303, 390-393).  The CRS SpMV is
// bound by the FP64 pipe: a warp issues an FP64 instruction (16 cycles of the
// SM) for the longest of its rows, 9 per lane where the LSCM rows have 7 on
// average.  Here the rows of one pass of a CTA (128) are sorted by length, so
// that a warp's rows are nearly equal, and stored so that its loads are
// coalesced.  Each lane still adds its row's terms in row_dot's order and the
// p.q sums keep their threads (rows return to them through shared memory), so
// results are bit-identical to the CRS kernels'.  Costs 12 bytes per nonzero
// and a pass over the matrix, once per matrix and layout.
//
// Measured on GB300, LSCM 808 x 808 (1.31 M rows, 18.3 M nonzeros): SpMV 62.8
// -> 53.3 us (4.6 TB/s), PCG iteration 111.1 -> 100.4 us.  Not used with other
// numbers of threads per row, where it loses: with one (the cotangent
// Laplacian, 4.2 M rows) sorting over 256 rows scatters the gathers of x and
// the SpMV takes 108 us instead of 91; with four or eight it is even; in FP32
// and double-float the FP64 pipe is not the bound (97 -> 112 us per mixed
// iteration).  A coalesced layout without the sorting was slower than CRS
// (68 us; one thread per row 104).
#include "nlgb_sell.h"

#include <algorithm>

namespace nlgb {
namespace {

constexpr int kSellWarps = kCTA / 32;
constexpr int kSellRows = kCTA / 2;     // rows of a pass

// One CTA per pass: row lengths per lane, ranks, slice widths, and the
// pass's place in the arrays (any order: a counter hands it out).
__global__ void __launch_bounds__(kCTA) k_sell_shape(int n, int tile_rows, int passes, const int* __restrict__ rp, uint2* shape, unsigned char* len,
                                                     unsigned char* perm, unsigned* ctl) {
  __shared__ int key[kCTA];
  __shared__ int sorted[kCTA];
  __shared__ unsigned base;
  constexpr int tpr = 2, rpp = kSellRows, rpw = 32 / tpr;
  const int t = threadIdx.x;
  const int tile = blockIdx.x / passes, pass = blockIdx.x % passes;
  const int b = tile * tile_rows + pass * rpp;
  const int hi = min(n, min((tile + 1) * tile_rows, b + rpp));
  const int rows = hi - b;
  int k = 0;
  if (t < rpp) {
    if (t < rows) {
      k = (rp[b + t + 1] - rp[b + t] + tpr - 1) / tpr;
      if (k > 255) { atomicOr(ctl + 1, 1u); k = 255; }
    }
    key[t] = k;
  }
  __syncthreads();
  if (t < rpp) {
    int rank = 0;
    for (int u = 0; u < rpp; ++u) rank += key[u] > k || (key[u] == k && u < t);
    sorted[rank] = t;
  }
  __syncthreads();
  if (t == 0) {
    unsigned w[kSellWarps], sum = 0;
    for (int i = 0; i < kSellWarps; ++i) {
      w[i] = (unsigned)key[sorted[i * rpw]];
      sum += w[i];
    }
    unsigned at = base = atomicAdd(ctl, sum);
    for (int i = 0; i < kSellWarps; ++i) {
      shape[(size_t)blockIdx.x * kSellWarps + i] = make_uint2(at, w[i]);
      at += w[i];
    }
  }
  if (t < rows) perm[b + t] = (unsigned char)sorted[t];
  // lane t of the pass: sorted row t / tpr, nonzeros t % tpr, t % tpr + tpr, ...
  const int r = sorted[t / tpr];
  const int nz = r < rows ? rp[b + r + 1] - rp[b + r] : 0;
  len[(size_t)blockIdx.x * kCTA + t] = (unsigned char)min(255, max(0, (nz - t % tpr + tpr - 1) / tpr));
}

__global__ void __launch_bounds__(kCTA) k_sell_fill(int n, int tile_rows, int passes, const int* __restrict__ rp,
                                                    const int* __restrict__ ci, const double* __restrict__ va,
                                                    const uint2* __restrict__ shape,
                                                    const unsigned char* __restrict__ len,
                                                    const unsigned char* __restrict__ perm, int* ci_out,
                                                    double* va_out) {
  const int t = threadIdx.x, lane = t & 31;
  const int tile = blockIdx.x / passes, pass = blockIdx.x % passes;
  const int b = tile * tile_rows + pass * kSellRows;
  const int hi = min(n, min((tile + 1) * tile_rows, b + kSellRows));
  const uint2 sh = shape[(size_t)blockIdx.x * kSellWarps + (t >> 5)];
  const int cnt = len[(size_t)blockIdx.x * kCTA + t];
  const int at = b + t / 2;
  const int src = at < hi ? rp[b + perm[at]] + t % 2 : 0;
  for (unsigned k = 0; k < sh.y; ++k) {
    const size_t o = ((size_t)sh.x + k) * 32 + lane;
    const bool in = (int)k < cnt;
    ci_out[o] = in ? ci[src + 2 * (int)k] : 0;
    va_out[o] = in ? va[src + 2 * (int)k] : 0.0;
  }
}

// A tile of q = A x: epi(row, q) by the thread that owns the row in the CRS
// kernels (thread 2 (row - base) of the pass starting at base).  The matrix is
// read once per SpMV: streaming loads leave L2 to the vectors.
template <typename Epi>
__device__ __forceinline__ void sell_tile(const SellView& m, int tile, int lo, int hi, const double* __restrict__ x,
                                          Epi&& epi) {
  __shared__ double sq[2][kSellRows];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = (int)threadIdx.x >> 1;
  size_t ps = (size_t)tile * m.passes;
  int buf = 0;
  for (int b = lo; b < hi; b += kSellRows, ++ps, buf ^= 1) {
    const uint2 sh = __ldg(m.shape + ps * kSellWarps + warp);
    const int n = __ldg(m.len + ps * kCTA + threadIdx.x);
    const bool mine = (threadIdx.x & 1) == 0 && b + sub < hi;
    const int to = mine ? __ldg(m.perm + b + sub) : 0;
    const int* c = m.ci + (size_t)sh.x * 32 + lane;
    const double* a = m.va + (size_t)sh.x * 32 + lane;
    const int w = (int)sh.y;
    double sum = 0.0;
#pragma unroll 4
    for (int k = 0; k < w; ++k) {
      const int cc = __ldcs(c + 32 * k);
      const double av = __ldcs(a + 32 * k);
      if (k < n) sum = fma(av, __ldg(x + cc), sum);
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    if (mine) sq[buf][to] = sum;
    __syncthreads();
    if (mine) epi(b + sub, sq[buf][sub]);
  }
}

// q = A p and the tile's p.q partial (k_spmv_pq<2>).
__global__ void __launch_bounds__(kCTA, 8) k_sell_pq(SysView s) {
  if (__ldcg(&s.st->status) != ST_RUNNING) return;
  const int tile = blockIdx.x, lo = tile_lo(s, tile), hi = tile_hi(s, tile);
  double acc[1] = {0.0};
  sell_tile(s.sell, tile, lo, hi, s.p, [&](int row, double q) {
    s.q[row] = q;
    acc[0] = fma(__ldcg(s.p + row), q, acc[0]);
  });
  block_sum<1>(acc);
  if (threadIdx.x == 0) __stcg(s.part + (size_t)tile * kParts + kSlotPQ, acc[0]);
}

// y = A x alone keeps the passes' barrier too: with warps running ahead of each
// other their gathers of x no longer meet in L1 (53 -> 73 us at 18.3 M nonzeros;
// slices dealt over the whole grid: 108 us).
__global__ void __launch_bounds__(kCTA, 8) k_sell_spmv(SellView m, int n, int tile_rows, const double* __restrict__ x,
                                                       double* __restrict__ y) {
  const int lo = blockIdx.x * tile_rows, hi = min(lo + tile_rows, n);
  sell_tile(m, blockIdx.x, lo, hi, x, [&](int row, double q) { y[row] = q; });
}

template <typename T>
bool try_alloc(T** p, size_t count, cudaStream_t s) {
  if (cudaMallocAsync(reinterpret_cast<void**>(p), std::max<size_t>(1, count) * sizeof(T), s) == cudaSuccess) return true;
  cudaGetLastError();
  *p = nullptr;
  return false;
}

bool suits(const DeviceCRS& A) {
  return A.owns && !A.lean && A.n > 0 && A.tpr == 2 && A.tile_rows > 0 && A.nnz >= kSellMinNnz &&
         A.nnz <= kSellMaxNnz;
}
long long most_elements(const DeviceCRS& A) { return A.nnz + A.nnz / 8; }
long long shape_ctas(int n, int tile_rows) {
  return (long long)((n + tile_rows - 1) / tile_rows) * ((tile_rows + kSellRows - 1) / kSellRows);
}
long long layout_bytes(int n, int tile_rows, long long elements) {
  return shape_ctas(n, tile_rows) * (kSellWarps * (long long)sizeof(uint2) + kCTA) + n + 12LL * elements;
}

}  // namespace

const void* sell_pq_kernel(const SysView& v) { return v.sell.va ? (const void*)k_sell_pq : nullptr; }

void sell_free(SellLayout& L, cudaStream_t s, bool async) {
  for (void* p : {(void*)L.shape, (void*)L.len, (void*)L.perm, (void*)L.ci, (void*)L.va})
    if (p) { if (async) cudaFreeAsync(p, s); else cudaFree(p); }
  L = SellLayout();
}

cudaError_t sell_prepare(DeviceCRS& A, SellView* view, cudaStream_t s, bool build) {
  *view = SellView{};
  std::lock_guard<std::mutex> lk(*A.lazy);
  if (!suits(A)) return cudaSuccess;
  SellLayout& L = A.sell;
  if (L.state != 0 && (L.tpr != A.tpr || L.tile_rows != A.tile_rows)) sell_free(L, s, true);
  auto hand_out = [&]() { *view = SellView{L.shape, L.len, L.perm, L.ci, L.va, L.passes}; };
  if (L.state != 0) {
    if (L.state > 0) hand_out();
    return cudaSuccess;
  }
  if (!build) return cudaSuccess;
  L.state = -1;
  L.tpr = A.tpr;
  L.tile_rows = A.tile_rows;
  L.passes = (A.tile_rows + kSellRows - 1) / kSellRows;
  const long long ctas = shape_ctas(A.n, A.tile_rows);
  unsigned* ctl = nullptr;
  if (ctas > (1LL << 30) || !try_alloc(&L.shape, (size_t)ctas * kSellWarps, s) ||
      !try_alloc(&L.len, (size_t)ctas * kCTA, s) || !try_alloc(&L.perm, (size_t)A.n, s) || !try_alloc(&ctl, 2, s))
    return cudaSuccess;   // no room: the CRS kernels run
  NLGB_CUDA_TRY(cudaMemsetAsync(ctl, 0, 2 * sizeof(unsigned), s));
  k_sell_shape<<<(unsigned)ctas, kCTA, 0, s>>>(A.n, A.tile_rows, L.passes, A.rp, L.shape, L.len, L.perm, ctl);
  count_launches(1);
  NLGB_CUDA_TRY(cudaGetLastError());
  unsigned h[2] = {0, 0};
  NLGB_CUDA_TRY(cudaMemcpyAsync(h, ctl, sizeof(h), cudaMemcpyDeviceToHost, s));
  NLGB_CUDA_TRY(cudaStreamSynchronize(s));
  NLGB_CUDA_TRY(cudaFreeAsync(ctl, s));
  // rows of more than 255 nonzeros per lane, or lengths so uneven within the
  // passes that padding adds more than an eighth: not worth it
  L.units = h[0];
  const size_t el = (size_t)L.units * 32;
  if (h[1] != 0 || (long long)el > most_elements(A) || !try_alloc(&L.ci, el, s) || !try_alloc(&L.va, el, s)) {
    sell_free(L, s, true);
    L.state = -1;
    L.tpr = A.tpr;
    L.tile_rows = A.tile_rows;
    return cudaSuccess;
  }
  k_sell_fill<<<(unsigned)ctas, kCTA, 0, s>>>(A.n, A.tile_rows, L.passes, A.rp, A.ci, A.va, L.shape, L.len, L.perm, L.ci,
                                              L.va);
  count_launches(1);
  NLGB_CUDA_TRY(cudaGetLastError());
  NLGB_CUDA_TRY(cudaStreamSynchronize(s));   // (another thread may use it on a stream of its own)
  L.state = 1;
  hand_out();
  return cudaSuccess;
}

long long sell_bytes(const DeviceCRS& A) {
  const SellLayout& L = A.sell;
  if (L.state <= 0) return 0;
  return layout_bytes(A.n, L.tile_rows, L.units * 32LL);
}

long long sell_most_bytes(const DeviceCRS& A) {
  return suits(A) ? layout_bytes(A.n, A.tile_rows, most_elements(A)) : 0;
}

cudaError_t sell_spmv64(const DeviceCRS& A, const SellView& m, const double* x, double* y, cudaStream_t s) {
  k_sell_spmv<<<(A.n + A.tile_rows - 1) / A.tile_rows, kCTA, 0, s>>>(m, A.n, A.tile_rows, x, y);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace nlgb
