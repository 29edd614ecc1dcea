// nlgb_persist.cu -- host side of the persistent PCG kernel (nlgb_persist.cuh):
// the tables of a matrix, the launch shapes, the launch.
#include "nlgb_persist.h"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>

namespace nlgb {
namespace {

constexpr int kPrepThreads = 512;

// ---------------------------------------------------------------------------
// Tables of one matrix (PersistLayout), one CTA per CTA of the solve.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kPrepThreads) k_persist_prep(int n, int R, int n_tiles, int C, int slots, int tpr,
                                                               int cluster, int stride,
                                                               const int* __restrict__ rp, const int* __restrict__ ci,
                                                               unsigned short* lci, unsigned short* perm, int* halo,
                                                               int* halo_n, int* most) {
  extern __shared__ unsigned words[];            // bitmap of the columns, then its exclusive counts
  __shared__ int sums[kPrepThreads];
  __shared__ int hist[65];
  const int per = n_tiles / C, extra = n_tiles % C, cta = (int)blockIdx.x;
  const int t0 = cta * per + min(cta, extra), cnt = per + (cta < extra ? 1 : 0);
  const int row0 = t0 * R, row1 = min(n, (t0 + cnt) * R), rows = row1 - row0, cap = slots * R;
  const int W = (n + 31) / 32;
  int* off = reinterpret_cast<int*>(words + W);
  for (int i = threadIdx.x; i < W; i += kPrepThreads) words[i] = 0u;
  for (int i = threadIdx.x; i < 65; i += kPrepThreads) hist[i] = 0;
  __syncthreads();
  const int k0 = rp[row0], k1 = rp[row1];
  for (int k = k0 + (int)threadIdx.x; k < k1; k += kPrepThreads) {
    const int c = ci[k];
    if (c < row0 || c >= row1) atomicOr(&words[c >> 5], 1u << (c & 31));
  }
  __syncthreads();
  // exclusive counts: each thread a run of words, then the runs in order
  const int run = (W + kPrepThreads - 1) / kPrepThreads;
  const int w0 = min(W, (int)threadIdx.x * run), w1 = min(W, w0 + run);
  int mine = 0;
  for (int w = w0; w < w1; ++w) mine += __popc(words[w]);
  sums[threadIdx.x] = mine;
  __syncthreads();
  for (int o = 1; o < kPrepThreads; o <<= 1) {
    const int t = (int)threadIdx.x >= o ? sums[threadIdx.x - o] : 0;
    __syncthreads();
    sums[threadIdx.x] += t;
    __syncthreads();
  }
  int at = sums[threadIdx.x] - mine;
  const int H = sums[kPrepThreads - 1];
  if (threadIdx.x == 0) {
    halo_n[cta] = H;
    atomicMax(most, H);
  }
  for (int w = w0; w < w1; ++w) {
    off[w] = at;
    unsigned b = words[w];
    while (b) {
      const int c = w * 32 + __ffs((int)b) - 1;
      b &= b - 1;
      if (at < stride) {
        int entry = c;
        if (cluster) {
          const int t = c / R, big = extra * (per + 1);
          const int rk = t < big ? t / (per + 1) : extra + (t - big) / per;
          entry = (rk << 16) | (c - (rk * per + min(rk, extra)) * R);
        }
        halo[(size_t)cta * stride + at] = entry;
      }
      ++at;
    }
  }
  __syncthreads();
  if (H > stride) return;                        // the matrix is not laid out
  for (int k = k0 + (int)threadIdx.x; k < k1; k += kPrepThreads) {
    const int c = ci[k];
    lci[k] = (unsigned short)(c >= row0 && c < row1
                                  ? c - row0
                                  : cap + off[c >> 5] + __popc(words[c >> 5] & ((1u << (c & 31)) - 1u)));
  }
  // rows by length (per lane), longest first
  for (int i = threadIdx.x; i < rows; i += kPrepThreads)
    atomicAdd(&hist[63 - min(63, (rp[row0 + i + 1] - rp[row0 + i] + tpr - 1) / tpr)], 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int b = 0; b < 64; ++b) { const int h = hist[b]; hist[b] = acc; acc += h; }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < rows; i += kPrepThreads) {
    const int b = 63 - min(63, (rp[row0 + i + 1] - rp[row0 + i] + tpr - 1) / tpr);
    perm[row0 + atomicAdd(&hist[b], 1)] = (unsigned short)i;
  }
}

const void* persist_kernel(int tpr, int mode, bool cluster, int nc) {
  return mode == kPersistDouble ? persist_kernel_f64(tpr, cluster, nc)
         : mode == kPersistDf   ? persist_kernel_df(tpr, cluster, nc)
                                : persist_kernel_mx(tpr, cluster, nc);
}

bool device_limits(int* sms, int* smem) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return true;
}

size_t smem_bytes(int slots, int R, int halo, size_t word) {
  return ((size_t)6 * slots * R + 2 * (size_t)halo) * word + (size_t)slots * 2 * kPersistRed * sizeof(double);
}

}  // namespace

int persist_ctas(const DeviceCRS& A, int n_tiles, int per_cta, int sms, int leave) {
  const bool alone = per_cta == kPersistAlone, rows_long = A.tpr > 2 && A.nnz > kPersistCluster * kPersistCtaNnz;
  int tiles = std::max(1, per_cta);
  if (A.tpr > 2) tiles = (int)std::max(1LL, std::min<long long>(tiles, kPersistCtaNnz * n_tiles / std::max(1LL, A.nnz)));
  const bool spread = alone && (A.tpr > 2 || (A.tpr == 2 && n_tiles > 2 * kPersistCluster));
  return persist_ctas_for(n_tiles, tiles, sms, leave, spread || rows_long);
}

int persist_ctas_for(int n_tiles, int per_cta, int sms, int leave, bool spread) {
  const int want = (n_tiles + per_cta - 1) / per_cta;
  if (n_tiles <= kPersistClusterTiles && (want <= kPersistCluster || !spread)) return std::min(want, kPersistCluster);
  const int ctas = std::min(want, sms - 1), fewer = sms - 1 - leave;
  if (leave == 0 || ctas <= fewer || fewer < 1) return ctas;
  const int slots = (n_tiles + fewer - 1) / fewer;
  return slots <= kPersistSlots ? (n_tiles + slots - 1) / slots : ctas;
}

double persist_iteration_us(int n_tiles, int ctas) {
  return 5.0 + 1.2 * (double)((n_tiles + ctas - 1) / std::max(1, ctas) - 1);   // (kSharedTiles' figures)
}

void PersistTables::release() {
  cudaFree(mem_);
  mem_ = nullptr;
  bytes_ = 0;
  lay_ = PersistLayout();
}

void PersistTables::release(cudaStream_t s) {
  if (mem_) cudaFreeAsync(mem_, s);
  mem_ = nullptr;
  release();
}

cudaError_t PersistTables::build(const DeviceCRS& A, int tile_rows, int n_tiles, cudaStream_t s, int per_cta,
                                 int leave) {
  int most = 0, *d = nullptr;
  NLGB_CUDA_TRY(cudaMallocAsync((void**)&d, sizeof(int), s));
  cudaError_t e = cudaMemsetAsync(d, 0, sizeof(int), s);
  if (e == cudaSuccess) e = begin(A, tile_rows, n_tiles, s, per_cta, d, leave);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&most, d, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFreeAsync(d, s);
  NLGB_CUDA_TRY(e);
  end(most, s);
  return cudaSuccess;
}

cudaError_t PersistTables::begin(const DeviceCRS& A, int tile_rows, int n_tiles, cudaStream_t s, int per_cta,
                                 int* most, int leave) {
  release();
  int sms = 0, smem_max = 0;
  if (A.n <= 0 || A.nnz <= 0 || A.n != A.m || tile_rows > 512 || !device_limits(&sms, &smem_max)) return cudaSuccess;
  const int ctas = persist_ctas(A, n_tiles, per_cta, sms, leave);
  if (ctas < 1) return cudaSuccess;
  cluster_ = ctas <= kPersistCluster && n_tiles <= kPersistClusterTiles;
  nnz_ = A.nnz;
  const int slots = (n_tiles + ctas - 1) / ctas;
  const int cap = slots * tile_rows;
  if (slots > kPersistSlots || cap > 8192) return cudaSuccess;
  const size_t W = (size_t)(A.n + 31) / 32;
  const size_t prep_smem = W * (sizeof(unsigned) + sizeof(int));
  if (prep_smem + 8192 > (size_t)smem_max) return cudaSuccess;
  // the halo the FP64 form has shared memory for (two words per entry)
  const size_t own = smem_bytes(slots, tile_rows, 0, sizeof(double));
  if (own + 8192 >= (size_t)smem_max) return cudaSuccess;
  const int stride = (int)std::min<size_t>(((size_t)smem_max - 8192 - own) / (2 * sizeof(double)), (size_t)A.n) & ~1;
  const size_t lci_b = ((size_t)A.nnz * sizeof(unsigned short) + 255) & ~(size_t)255;
  const size_t perm_b = ((size_t)A.n * sizeof(unsigned short) + 255) & ~(size_t)255;
  const size_t halo_b = ((size_t)ctas * std::max(1, stride) * sizeof(int) + 255) & ~(size_t)255;
  const size_t bytes = lci_b + perm_b + halo_b + (size_t)ctas * sizeof(int);
  const cudaError_t room = cudaMallocAsync(&mem_, bytes, s);
  if (room == cudaErrorMemoryAllocation) {       // the other executors need no tables
    cudaGetLastError();
    mem_ = nullptr;
    return cudaSuccess;
  }
  NLGB_CUDA_TRY(room);
  bytes_ = bytes;
  char* m = static_cast<char*>(mem_);
  unsigned short* lci = reinterpret_cast<unsigned short*>(m);
  unsigned short* perm = reinterpret_cast<unsigned short*>(m + lci_b);
  int* halo = reinterpret_cast<int*>(m + lci_b + perm_b);
  int* halo_n = reinterpret_cast<int*>(m + lci_b + perm_b + halo_b);
  NLGB_CUDA_TRY(cudaFuncSetAttribute((const void*)k_persist_prep, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     smem_max - 8192));
  k_persist_prep<<<ctas, kPrepThreads, prep_smem, s>>>(A.n, tile_rows, n_tiles, ctas, slots, A.tpr, cluster_ ? 1 : 0,
                                                       stride, A.rp, A.ci, lci, perm, halo, halo_n, most);
  count_launches(1);
  NLGB_CUDA_TRY(cudaGetLastError());
  lay_.slots = slots;
  lay_.halo_stride = stride;
  ctas_ = ctas;
  lay_.lci = lci;
  lay_.perm = perm;
  lay_.halo = halo;
  lay_.halo_n = halo_n;
  return cudaSuccess;
}

void PersistTables::end(int most, cudaStream_t s) {
  if (!mem_) return;
  if (most > lay_.halo_stride) {
    release(s);
    return;
  }
  lay_.halo_cap = (most + 1) & ~1;
  lay_.ctas = ctas_;
}

PersistPlan PersistTables::plan(int tile_rows, int tpr, int mode) const {
  PersistPlan p;
  int sms = 0, smem_max = 0, dev = 0, l2 = 0;
  if (!usable() || !device_limits(&sms, &smem_max) || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess)
    return p;
  // values and columns within L2: one CTA per SM cannot stream them from HBM (us
  // per FP64 iteration, cooperative kernel -> this: 126 MB 92.9 -> 81.2, 142 MB
  // 84.6 -> 91.5, 152 MB 99.4 -> 107.8, 208 MB 110.4 -> 130.2; mixed, graph ->
  // this: 114 MB 72.7 -> 53.9, 139 MB 83.9 -> 109.9)
  if (nnz_ * (mode == kPersistMixed ? 8 : 12) > (long long)l2) return p;
  // 256 threads where they hold every row in registers, else 512
  const int per_lane_rows = (lay_.slots * tile_rows * tpr + 255) / 256;
  p.cluster = cluster_;
  p.block = per_lane_rows <= 1 ? 256 : kPersistBlock;
  p.grid = lay_.ctas + (cluster_ ? 0 : 1);
  const int nc = p.block == 256 ? 1 : (per_lane_rows + 1) / 2;
  const size_t word = mode == kPersistMixed ? sizeof(float) : sizeof(double);
  p.smem = (int)smem_bytes(lay_.slots, tile_rows, lay_.halo_cap, word);
  p.kernel = persist_kernel(tpr, mode, cluster_, nc);
  const void* fn = p.kernel;
  bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max - 8192) == cudaSuccess;
  if (ok && cluster_) {
    ok = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    if (ok) {
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute at;
      std::memset(&cfg, 0, sizeof(cfg));
      std::memset(&at, 0, sizeof(at));
      cfg.gridDim = dim3((unsigned)p.grid);
      cfg.blockDim = dim3((unsigned)p.block);
      cfg.dynamicSmemBytes = (size_t)p.smem;
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = (unsigned)p.grid;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      int nc = 0;
      ok = cudaOccupancyMaxActiveClusters(&nc, fn, &cfg) == cudaSuccess && nc >= 1;
    }
  } else if (ok) {
    int per_sm = 0;
    ok = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, p.block, (size_t)p.smem) == cudaSuccess && per_sm >= 1;
  }
  if (!ok) cudaGetLastError();
  p.usable = ok;
  return p;
}

cudaError_t persist_launch(const PersistPlan& p, const PersistArgs& args, cudaStream_t s) {
  PersistArgs a = args;
  a.wait_ns = 4000000000ULL;
  if (const char* t = std::getenv("NLGB_BARRIER_TIMEOUT_MS"))
    if (const double ms = std::atof(t); ms > 0.0) a.wait_ns = (unsigned long long)(ms * 1e6);
  if (const char* t = std::getenv("NLGB_TEST_PERSIST_REFUSE")) {
    static std::atomic<long long> asked{0};
    if (++asked >= std::atoll(t)) {
      set_error("persistent kernel: launch refused (NLGB_TEST_PERSIST_REFUSE)");
      return cudaErrorCooperativeLaunchTooLarge;
    }
  }
  const char* shortfall = p.cluster ? nullptr : std::getenv("NLGB_TEST_PERSIST_SHORTFALL");
  void* params[] = {&a};
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  std::memset(&cfg, 0, sizeof(cfg));
  std::memset(&at, 0, sizeof(at));
  cfg.gridDim = dim3((unsigned)(shortfall && shortfall[0] == '1' ? a.lay.ctas : p.grid));
  cfg.blockDim = dim3((unsigned)p.block);
  cfg.dynamicSmemBytes = (size_t)p.smem;
  cfg.stream = s;
  if (p.cluster) {
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)p.grid;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
  } else {
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
  }
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  NLGB_CUDA_TRY(cudaLaunchKernelExC(&cfg, p.kernel, params));
  count_launches(1);
  return cudaSuccess;
}

}  // namespace nlgb
