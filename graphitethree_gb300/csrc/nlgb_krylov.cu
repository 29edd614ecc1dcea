// nlgb_krylov.cu -- Krylov solvers for general square systems: BiCGSTAB and
// restarted GMRES(m), FP64, with Jacobi (or no) right preconditioning.
//
// Reference context: OpenNL's NL_BICGSTAB and NL_GMRES solvers, selected
// through nlSolverParameteri(NL_SOLVER, ...) or nlSolveSystemIterative
// (src/lib/OGF/scene_graph/NL/matrix.cpp:390-393), used by the WarpDrive /
// optimal-transport Newton steps
// (plugins/OGF/WarpDrive/commands/mesh_grob_transport_commands.cpp:456-474),
// whose Jacobians are not symmetric.  Published algorithms restated here:
// BiCGSTAB, H. A. van der Vorst, SIAM J. Sci. Stat. Comput. 13 (1992);
// GMRES(m), Y. Saad & M. H. Schultz, SIAM J. Sci. Stat. Comput. 7 (1986),
// with Givens rotations and classical Gram-Schmidt applied twice (CGS2; as
// stable as modified Gram-Schmidt in practice, L. Giraud, J. Langou &
// M. Rozloznik 2005) so that an inner step needs two multi-dot passes
// instead of 2(j + 1) dependent dot/axpy passes.
//
// Layout: the matrix's own tiles (DeviceCRS::tile_rows, threads per row);
// every dot product is a set of per-tile partials reduced in a fixed order
// by one CTA (canon_reduce), and every scalar step runs on the device, so the
// host only enqueues kernels and polls the status once per chunk (BiCGSTAB)
// or per restart cycle (GMRES).  BiCGSTAB's scalar steps run in the prologue
// of the vector kernel that uses them.  Kernels return at once when the system is no
// longer running, which makes overshooting a chunk harmless.
#include "nlgb_core.cuh"
#include "nlgb_internal.h"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace nlgb {
namespace {

constexpr int kMaxRestart = 64;     // GMRES(m): m <= 64
constexpr int kChunk = 16;          // BiCGSTAB iterations between status polls

struct KrState {
  double alpha, omega, beta;        // BiCGSTAB scalars (beta: GMRES too)
  double rho[2];                    // by the parity of the iteration that uses it
  double bnorm2, thresh2, rr, rr_true;
  double gnorm;                     // GMRES: |g_{j+1}| (residual estimate)
  long long iter, max_iter;
  int status;                       // ST_*
  int zero_rhs;
  int j;                            // GMRES: inner step of the cycle
  int cyc_done;                     // GMRES: this cycle is finished
  int m;                            // GMRES restart length
  int pad_;
  double H[(kMaxRestart + 1) * kMaxRestart];   // column-major, (m + 1) x m
  double cs[kMaxRestart], sn[kMaxRestart], g[kMaxRestart + 1], y[kMaxRestart];
  int act[kMaxRestart + 1];         // GMRES: step j of this cycle is to be run
};

struct KrView {
  int n, tile_rows, n_tiles;
  const int* rp;
  const int* ci;
  const double* va;
  const double* dinv;
  double* part;      // n_tiles * kParts
  KrState* st;
  double* mpart;     // GMRES: per CTA of a step kernel m + 1 multi-dot partials, then its w.w
  int mstride;
  int step_ctas, step_rows;   // CTAs of the step kernels and rows of each
};

__device__ __forceinline__ bool running(const KrView& v) {
  return *((volatile int*)&v.st->status) == ST_RUNNING;
}
__device__ __forceinline__ int step_lo(const KrView& v) { return (int)blockIdx.x * v.step_rows; }
__device__ __forceinline__ int step_hi(const KrView& v) { return min(v.n, ((int)blockIdx.x + 1) * v.step_rows); }
__device__ __forceinline__ int lo_of(const KrView& v) { return blockIdx.x * v.tile_rows; }
__device__ __forceinline__ int hi_of(const KrView& v) { return min(v.n, (int)(blockIdx.x + 1) * v.tile_rows); }

template <int K>
__device__ __forceinline__ void put_tile(const KrView& v, int slot, double (&a)[K]) {
  block_sum<K>(a);
  if (threadIdx.x == 0)
    for (int k = 0; k < K; ++k) v.part[(size_t)blockIdx.x * kParts + slot + k] = a[k];
}

template <int K>
__device__ __forceinline__ void sums(const KrView& v, int slot, double (&o)[K]) {
  int comp[K];
  for (int k = 0; k < K; ++k) comp[k] = slot + k;
  canon_reduce<K>(v.part, v.n_tiles, comp, o);
}

__device__ __forceinline__ bool finite_nz(double x) { return x == x && x != 0.0 && fabs(x) < 1e300; }

// y = A x on this CTA's tile, epi(row, (A x)_row) by the row's lane 0.
template <int T, typename Epi>
__device__ __forceinline__ void tile_spmv(const KrView& v, const double* x, Epi&& epi) {
  tile_rows_dot<T, double, double, double, false>(v.rp, v.ci, v.va, x, lo_of(v), hi_of(v), epi);
}

// ---------------------------------------------------------------------------
// BiCGSTAB (right preconditioning, M^-1 = D^-1):
//   r = b - A x, rh = r, rho = rh.r, p = v = 0, alpha = omega = 1
//   loop: p = r + beta (p - omega v); y = M^-1 p; v = A y; alpha = rho / rh.v
//         s = r - alpha v; z = M^-1 s; t = A z; omega = t.s / t.t
//         x += alpha y + omega z; r = s - omega t
//         stop on ||r|| <= eps ||b||; beta = (rh.r / rho)(alpha / omega)
// Vectors: r (holds s after the alpha step), rh, p, v, y, z, t.
// ---------------------------------------------------------------------------
struct BiVecs { const double* b; double *x, *r, *rh, *p, *v, *y, *z, *t; };

template <int T>
__global__ void __launch_bounds__(kCTA) k_bi_init(KrView v, BiVecs w) {
  double a[2] = {0.0, 0.0};
  tile_spmv<T>(v, w.x, [&](int i, double ax) {
    const double bi = w.b[i], ri = bi - ax;
    w.r[i] = ri; w.rh[i] = ri; w.p[i] = 0.0; w.v[i] = 0.0;
    a[0] = fma(bi, bi, a[0]);
    a[1] = fma(ri, ri, a[1]);
  });
  put_tile<2>(v, 0, a);
}

__global__ void k_bi_init_scalar(KrView v) {
  double o[2];
  sums<2>(v, 0, o);
  if (threadIdx.x != 0) return;
  KrState* st = v.st;
  st->bnorm2 = o[0];
  st->rr = o[1];
  st->rho[0] = o[1];            // rh = r
  st->alpha = st->omega = 1.0;
  st->beta = o[1];              // (rho / 1) (1 / 1); p = r on the first step
  if (!(o[0] > 0.0)) { st->zero_rhs = o[0] == 0.0; st->status = o[0] == 0.0 ? ST_CONVERGED : ST_BREAKDOWN; return; }
  if (o[1] <= st->thresh2 * o[0]) { st->status = ST_CONVERGED; return; }
  if (st->max_iter <= 0) { st->status = ST_MAX_ITER; return; }
  st->status = ST_RUNNING;
}

// The vector kernels of the iteration (p, s, x/r): CTAs of 1024 threads, one
// per SM, or of 256 up to kBiSmall rows per SM.  Each reduces the partials of
// the SpMV or update before it in its prologue and takes the scalar step
// itself; CTA 0 also writes the scalars to the state, where only later kernels
// read them (rho alternates between two slots; a status that turns while a CTA
// starts tells it to return, which its own step would).  As one-CTA kernels
// between the vector kernels the three scalar steps took 28 of the 129 us of an
// iteration on 1024 x 1024 unknowns; 120 us now.  One CTA per SM, because the
// reduction costs each CTA about 1,000 cycles of the SM's FP64 pipe: three CTAs
// of 512 threads 134 us, six of 256 140.  With few rows a CTA of 256 threads
// starts and synchronises sooner (us per iteration, before, 256, 1024 threads):
// 235 x 142 59.2, 51.2, 62.2; 400 x 380 65.0, 56.5, 65.4; 700 x 650 88.3, 75.0,
// 81.8; 1024 x 1024 129.1, 122.2, 119.6.
constexpr int kBiThreads = 1024;
constexpr int kBiQuarters = kBiThreads / kCTA;
constexpr int kBiSmall = 4096;

// The sums of the tiles' partials (canon_reduce's order), in every thread.
template <int K>
__device__ __forceinline__ void wide_sums(const KrView& v, int slot, double (&o)[K]) {
  __shared__ double red[K][kStage];
  __shared__ double tot[K];
  const int t = threadIdx.x;
  if (t < kCTA) {
#pragma unroll
    for (int k = 0; k < K; ++k) o[k] = 0.0;
#pragma unroll 8
    for (int i = t; i < v.n_tiles; i += kCTA)
#pragma unroll
      for (int k = 0; k < K; ++k) o[k] += __ldcg(v.part + (size_t)i * kParts + slot + k);
#pragma unroll
    for (int k = 0; k < K; ++k) red[k][stage_at(t)] = o[k];
  }
  __syncthreads();
  if (t < 32 * K) {
    const double s = stage_sum(red[t >> 5]);
    if ((t & 31) == 0) tot[t >> 5] = s;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) o[k] = tot[k];
}

// load and body over rows lo, lo + stride, ... < hi: U rows of a thread in flight.
template <int U, int N, typename Load, typename Body>
__device__ __forceinline__ void rows_in_flight(int lo, int hi, int stride, Load&& load, Body&& body) {
  for (int i = lo; i < hi; i += U * stride) {
    double a[U][N];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u * stride < hi) load(i + u * stride, a[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u * stride < hi) body(i + u * stride, a[u]);
  }
}

// The same answer in every thread, also while CTA 0 writes the status.
__device__ __forceinline__ bool stopped(const KrView& v) { return __syncthreads_or(!running(v)) != 0; }

// The end of iteration it (its r.r and rh.r): the stopping tests and beta.
__device__ __forceinline__ int bi_end(const KrView& v, long long it, double rr, double rho, bool write, double* beta) {
  KrState* st = v.st;
  const double alpha = st->alpha, omega = st->omega, rho0 = st->rho[it & 1];
  int status = ST_RUNNING;
  if (!(rr <= 1e300)) status = ST_BREAKDOWN;
  else if (rr <= st->thresh2 * st->bnorm2) status = ST_CONVERGED;
  else if (it + 1 >= st->max_iter) status = ST_MAX_ITER;
  else if (!finite_nz(rho) || !finite_nz(omega)) status = ST_BREAKDOWN;
  else *beta = (rho / rho0) * (alpha / omega);
  if (write) {
    st->iter = it + 1;
    st->rr = rr;
    if (status == ST_RUNNING) st->rho[(it + 1) & 1] = rho;
    else st->status = status;
  }
  return status;
}

// fold: the end of iteration it - 1 first.
__global__ void __launch_bounds__(kBiThreads, 1) k_bi_p(KrView v, BiVecs w, long long it, int fold) {
  if (stopped(v)) return;
  double beta, omega = v.st->omega;
  if (fold) {
    double o[2];
    wide_sums<2>(v, 3, o);
    if (bi_end(v, it - 1, o[0], o[1], blockIdx.x == 0 && threadIdx.x == 0, &beta) != ST_RUNNING) return;
  } else {
    beta = v.st->beta;
  }
  rows_in_flight<4, 4>(step_lo(v) + (int)threadIdx.x, step_hi(v), (int)blockDim.x,
    [&](int i, double (&a)[4]) { a[0] = w.r[i]; a[1] = w.p[i]; a[2] = w.v[i]; a[3] = __ldg(v.dinv + i); },
    [&](int i, double (&a)[4]) {
      const double pi = a[0] + beta * (a[1] - omega * a[2]);
      w.p[i] = pi;
      w.y[i] = a[3] * pi;
    });
}

template <int T>
__global__ void __launch_bounds__(kCTA, 8) k_bi_v(KrView v, BiVecs w) {
  if (!running(v)) return;
  double a[1] = {0.0};
  tile_spmv<T>(v, w.y, [&](int i, double q) { w.v[i] = q; a[0] = fma(w.rh[i], q, a[0]); });
  put_tile<1>(v, 0, a);
}

__global__ void __launch_bounds__(kBiThreads, 1) k_bi_s(KrView v, BiVecs w, long long it) {
  if (stopped(v)) return;
  double o[1];
  wide_sums<1>(v, 0, o);
  const bool ok = finite_nz(o[0]);
  const double alpha = v.st->rho[it & 1] / o[0];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (ok) v.st->alpha = alpha;
    else v.st->status = ST_BREAKDOWN;
  }
  if (!ok) return;
  rows_in_flight<4, 3>(step_lo(v) + (int)threadIdx.x, step_hi(v), (int)blockDim.x,
    [&](int i, double (&a)[3]) { a[0] = w.r[i]; a[1] = w.v[i]; a[2] = __ldg(v.dinv + i); },
    [&](int i, double (&a)[3]) {
      const double si = a[0] - alpha * a[1];
      w.r[i] = si;                      // r now holds s
      w.z[i] = a[2] * si;
    });
}

template <int T>
__global__ void __launch_bounds__(kCTA, 8) k_bi_t(KrView v, BiVecs w) {
  if (!running(v)) return;
  double a[2] = {0.0, 0.0};
  tile_spmv<T>(v, w.z, [&](int i, double q) {
    w.t[i] = q;
    a[0] = fma(q, w.r[i], a[0]);      // t.s
    a[1] = fma(q, q, a[1]);           // t.t
  });
  put_tile<2>(v, 1, a);
}

// Each quarter of the CTA (256 threads, a barrier of its own) takes a tile.
__global__ void __launch_bounds__(kBiThreads, 1) k_bi_xr(KrView v, BiVecs w) {
  if (!running(v)) return;
  __shared__ double red[kBiQuarters][2][kStage];
  double o[2];
  wide_sums<2>(v, 1, o);
  const double alpha = v.st->alpha, omega = o[1] > 0.0 ? o[0] / o[1] : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) v.st->omega = omega;
  const int quarters = (int)blockDim.x / kCTA, qd = threadIdx.x / kCTA, t = threadIdx.x % kCTA;
  for (int tile = (int)blockIdx.x * quarters + qd; tile < v.n_tiles; tile += (int)gridDim.x * quarters) {
    const int lo = tile * v.tile_rows, hi = min(v.n, lo + v.tile_rows);
    double rr = 0.0, rhr = 0.0;
    rows_in_flight<2, 6>(lo + t, hi, kCTA,
      [&](int i, double (&a)[6]) {
        a[0] = w.x[i]; a[1] = w.y[i]; a[2] = w.z[i]; a[3] = w.r[i]; a[4] = w.t[i]; a[5] = w.rh[i];
      },
      [&](int i, double (&a)[6]) {
        w.x[i] = a[0] + (alpha * a[1] + omega * a[2]);
        const double ri = a[3] - omega * a[4];
        w.r[i] = ri;
        rr = fma(ri, ri, rr);
        rhr = fma(a[5], ri, rhr);
      });
    red[qd][0][stage_at(t)] = rr;
    red[qd][1][stage_at(t)] = rhr;
    asm volatile("bar.sync %0, %1;" ::"r"(1 + qd), "n"(kCTA) : "memory");
    if (t < 64) {
      const double s = stage_sum(red[qd][t >> 5]);
      if ((t & 31) == 0) v.part[(size_t)tile * kParts + 3 + (t >> 5)] = s;
    }
    asm volatile("bar.sync %0, %1;" ::"r"(1 + qd), "n"(kCTA) : "memory");   // red[qd] is free again
  }
}

// Before a poll: the end of iteration it, for the host and for a k_bi_p without it.
__global__ void __launch_bounds__(kBiThreads, 1) k_bi_end(KrView v, long long it) {
  if (!running(v)) return;
  double o[2], beta = 0.0;
  wide_sums<2>(v, 3, o);
  if (threadIdx.x == 0 && bi_end(v, it, o[0], o[1], true, &beta) == ST_RUNNING) v.st->beta = beta;
}

// True residual ||b - A x||^2 of the returned x (and x = 0 when b = 0).
template <int T>
__global__ void __launch_bounds__(kCTA) k_kr_true(KrView v, const double* b, double* x) {
  double a[1] = {0.0};
  if (v.st->zero_rhs) {
    for (int i = lo_of(v) + threadIdx.x; i < hi_of(v); i += kCTA) x[i] = 0.0;
  } else {
    tile_spmv<T>(v, x, [&](int i, double ax) { const double ri = b[i] - ax; a[0] = fma(ri, ri, a[0]); });
  }
  put_tile<1>(v, 6, a);
}

__global__ void k_kr_true_scalar(KrView v) {
  double o[1];
  sums<1>(v, 6, o);
  if (threadIdx.x == 0) v.st->rr_true = o[0];
}

// ---------------------------------------------------------------------------
// GMRES(m) (right preconditioning, M^-1 = D^-1), one cycle:
//   r = b - A x, beta = ||r||, V0 = r / beta, g = beta e1
//   for j < m: w = A M^-1 V_j; classical Gram-Schmidt against V_0..V_j,
//              twice (CGS2: h = V^T w, w -= V h; again; H_j = h + h2);
//              H_{j+1,j} = ||w||, V_{j+1} = w / H_{j+1,j}; Givens rotations
//              on column j, g; |g_{j+1}| is the residual norm
//   y = H^-1 g (upper triangular), x += M^-1 (V y)
// Convergence is decided on the true residual at the start of a cycle.
// ---------------------------------------------------------------------------
struct GmVecs { const double* b; double* x; double* V; double* u; size_t ld; };

template <int T>
__global__ void __launch_bounds__(kCTA) k_gm_residual(KrView v, GmVecs w) {
  if (*((volatile int*)&v.st->status) != ST_RUNNING) return;
  double a[2] = {0.0, 0.0};
  tile_spmv<T>(v, w.x, [&](int i, double ax) {
    const double bi = w.b[i], ri = bi - ax;
    w.V[i] = ri;
    a[0] = fma(bi, bi, a[0]);
    a[1] = fma(ri, ri, a[1]);
  });
  put_tile<2>(v, 0, a);
}

__global__ void k_gm_start(KrView v, int first) {
  if ((int)threadIdx.x <= kMaxRestart) v.st->act[threadIdx.x] = 0;   // no step of this cycle yet
  if (*((volatile int*)&v.st->status) != ST_RUNNING) return;
  double o[2];
  sums<2>(v, 0, o);                // (synchronises the CTA)
  if (threadIdx.x != 0) return;
  KrState* st = v.st;
  if (first) {
    st->bnorm2 = o[0];
    if (!(o[0] > 0.0)) { st->zero_rhs = o[0] == 0.0; st->status = o[0] == 0.0 ? ST_CONVERGED : ST_BREAKDOWN; return; }
  }
  st->rr = o[1];
  if (!(o[1] <= 1e300)) { st->status = ST_BREAKDOWN; return; }
  if (o[1] <= st->thresh2 * st->bnorm2) { st->status = ST_CONVERGED; return; }
  if (st->iter >= st->max_iter) { st->status = ST_MAX_ITER; return; }
  const double beta = sqrt(o[1]);
  for (int k = 0; k <= st->m; ++k) st->g[k] = 0.0;
  st->g[0] = beta;
  st->gnorm = beta;
  st->j = 0;
  st->cyc_done = 0;
  st->beta = beta;
  st->act[0] = 1;
}

// A step of a cycle is four kernels of one 512-thread CTA per SM (ten
// launches over the matrix's tiles before):
//   k_gm_spmv    w = A u, and the partials of h = V^T w;
//   k_gm_orth    h summed by every CTA, w -= V h, partials of h2 = V^T w;
//   k_gm_orth    h2 summed, w -= V h2, partials of w.w;
//   k_gm_next    the norm, V_{j+1} = w / ||w||, u = M^-1 V_{j+1}; one more CTA
//                turns column j of H into the QR factors and decides whether
//                the cycle goes on.
// V fits L2 up to about 16 M entries; the FP64 pipe bounds the rest: 4 n (j + 1)
// products per step, 32 of the 98 us a step takes at 314,323 rows (j = 15 on
// average).  What was slow before: a block sum per coefficient and tile of 384
// rows cost three times its products (67 us per round), and the reductions and
// the norm were kernels of one CTA.  Measured on GB300, convection-diffusion
// 601 x 523, GMRES(30): 231 -> 98 us per step (with 1,024 threads 108: a
// group's eight sums cost every warp nine FP64 instructions, 2.4 us of the SM
// with 32 warps).
constexpr int kGmThreads = 512;
constexpr int kGmWarps = kGmThreads / 32;

// Sums of eight per-lane values over the warp: lane l returns value
// (l / 4) mod 8 (the lanes that carry a value halve at each level, so eight
// sums take nine additions).
__device__ __forceinline__ double warp_sum8(const double (&a)[8]) {
  const int l = threadIdx.x & 31;
  double u[4], t[2];
#pragma unroll
  for (int q = 0; q < 4; ++q)
    u[q] = ((l & 16) ? a[q + 4] : a[q]) + __shfl_xor_sync(0xffffffffu, (l & 16) ? a[q] : a[q + 4], 16);
#pragma unroll
  for (int q = 0; q < 2; ++q)
    t[q] = ((l & 8) ? u[q + 2] : u[q]) + __shfl_xor_sync(0xffffffffu, (l & 8) ? u[q] : u[q + 2], 8);
  double s = ((l & 4) ? t[1] : t[0]) + __shfl_xor_sync(0xffffffffu, (l & 4) ? t[0] : t[1], 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}

__device__ __forceinline__ bool step_active(const KrView& v, int j) { return *((volatile int*)&v.st->act[j]) != 0; }

// This CTA's partials of V_i . w, i <= j (every thread calls it).
__device__ __forceinline__ void step_dots(const KrView& v, const GmVecs& w, const double* wn, int j) {
  __shared__ double red[kGmWarps][kMaxRestart + 1];
  const int lo = step_lo(v), hi = step_hi(v), warp = threadIdx.x >> 5, l = threadIdx.x & 31;
  for (int i0 = 0; i0 <= j; i0 += 8) {
    double a[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const int c = min(8, j + 1 - i0);
    const double* Vi = w.V + (size_t)i0 * w.ld;
    for (int r = lo + (int)threadIdx.x; r < hi; r += kGmThreads) {
      const double x = wn[r];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < c) a[q] = fma(x, Vi[(size_t)q * w.ld + r], a[q]);
    }
    const double s = warp_sum8(a);
    if ((l & 3) == 0 && (l >> 2) < c) red[warp][i0 + (l >> 2)] = s;
  }
  __syncthreads();
  // eight lanes per coefficient
  const int i = threadIdx.x >> 3, p = threadIdx.x & 7;
  double s = 0.0;
  if (i <= j) {
    s = red[p][i];
#pragma unroll
    for (int k = 1; k < kGmWarps / 8; ++k) s += red[p + 8 * k][i];
  }
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  if (i <= j && p == 0) v.mpart[(size_t)blockIdx.x * v.mstride + i] = s;
}

// The coefficients i <= j summed over the CTAs into h (shared memory).
__device__ __forceinline__ void step_sums(const KrView& v, int j, double* h) {
  const int l = threadIdx.x & 31;
  for (int i = threadIdx.x >> 5; i <= j; i += kGmWarps) {
    double s = 0.0;
    for (int g = l; g < v.step_ctas; g += 32) s += v.mpart[(size_t)g * v.mstride + i];
    s = warp_sum(s);
    if (l == 0) h[i] = s;
  }
  __syncthreads();
}

// V_0 = r / ||r||, u = M^-1 V_0 (prec 0: a general preconditioner follows).
__global__ void k_gm_scale0(KrView v, GmVecs w, int prec) {
  if (!step_active(v, 0)) return;
  const double inv = 1.0 / v.st->beta;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < v.n; i += (long long)gridDim.x * blockDim.x) {
    const double x = w.V[i] * inv;
    w.V[i] = x;
    if (prec) w.u[i] = v.dinv[i] * x;
  }
}

template <int T>
__global__ void __launch_bounds__(kGmThreads, 1) k_gm_spmv(KrView v, GmVecs w, int j) {
  if (!step_active(v, j)) return;
  double* Wn = w.V + (size_t)(j + 1) * w.ld;
  const int lo = step_lo(v), hi = step_hi(v);
  constexpr int RPP = kGmThreads / T;
  for (int base = lo; base < hi; base += RPP) {
    const int row = base + (int)threadIdx.x / T, lane = threadIdx.x % T;
    // (row_dot with up to eight nonzeros per lane in flight: one CTA per SM
    // hides less latency than the tiles' eight)
    double q = 0.0;
    if (row < hi) {
      const int k1 = __ldg(v.rp + row + 1);
      for (int k = __ldg(v.rp + row) + lane; k < k1; k += 8 * T) {
        double x[8], a[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (k + u * T < k1) {
            x[u] = __ldg(w.u + __ldg(v.ci + k + u * T));
            a[u] = __ldg(v.va + k + u * T);
          }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (k + u * T < k1) q = fma(a[u], x[u], q);
      }
    }
    q = subwarp_sum<T, double>(q);
    if (row < hi && lane == 0) Wn[row] = q;
  }
  __syncthreads();
  step_dots(v, w, Wn, j);
}

// One Gram-Schmidt round: the sums of the partials, w -= V h (i in order);
// then the second round's partials, or after it (round 1) those of w.w.
__global__ void __launch_bounds__(kGmThreads, 1) k_gm_orth(KrView v, GmVecs w, int j, int round, const double* pin) {
  if (!step_active(v, j)) return;
  __shared__ double h[kMaxRestart + 1];
  __shared__ double rr[kGmWarps];
  {
    KrView in = v;
    in.mpart = const_cast<double*>(pin);
    step_sums(in, j, h);
  }
  if (blockIdx.x == 0 && (int)threadIdx.x <= j) {
    double* Hj = v.st->H + j * (kMaxRestart + 1);
    Hj[threadIdx.x] = round == 0 ? h[threadIdx.x] : Hj[threadIdx.x] + h[threadIdx.x];
  }
  double* Wn = w.V + (size_t)(j + 1) * w.ld;
  const int lo = step_lo(v), hi = step_hi(v);
  double a = 0.0;
  for (int r = lo + (int)threadIdx.x; r < hi; r += kGmThreads) {
    double x = Wn[r];
#pragma unroll 8
    for (int i = 0; i <= j; ++i) x -= h[i] * w.V[(size_t)i * w.ld + r];
    Wn[r] = x;
    a = fma(x, x, a);
  }
  if (round == 0) {
    step_dots(v, w, Wn, j);      // (each thread reads back its own rows)
    return;
  }
  a = warp_sum(a);
  if ((threadIdx.x & 31) == 0) rr[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x < 32) {
    a = warp_sum((int)threadIdx.x < kGmWarps ? rr[threadIdx.x] : 0.0);
    if (threadIdx.x == 0) v.mpart[(size_t)blockIdx.x * v.mstride] = a;
  }
}

// H_{j+1,j} = ||w||, V_{j+1} = w / it, u = M^-1 V_{j+1}; Givens rotations and
// cycle control by the last CTA.
__global__ void __launch_bounds__(kGmThreads, 1) k_gm_next(KrView v, GmVecs w, int j, int prec) {
  if (!step_active(v, j)) return;
  __shared__ double nrm[1], rotated;
  __shared__ double hc[kMaxRestart + 1], cs[kMaxRestart], sn[kMaxRestart];
  KrState* st = v.st;
  double* Hj = st->H + j * (kMaxRestart + 1);
  const bool last = blockIdx.x == gridDim.x - 1;   // no rows: column j and the rotations
  if (last) {
    if ((int)threadIdx.x <= j) {
      hc[threadIdx.x] = Hj[threadIdx.x];
      if ((int)threadIdx.x < j) { cs[threadIdx.x] = st->cs[threadIdx.x]; sn[threadIdx.x] = st->sn[threadIdx.x]; }
    }
    __syncthreads();
    if (threadIdx.x == 32) {                       // the previous rotations, while warp 0 sums
      double a = hc[0];
      for (int k = 0; k < j; ++k) {
        const double b = hc[k + 1], c = cs[k], s = sn[k];
        const double up = c * a + s * b;
        Hj[k] = up;
        a = -s * a + c * b;
      }
      rotated = a;
    }
  }
  step_sums(v, 0, nrm);
  const double hn = sqrt(nrm[0]);
  if (!last) {
    if (hn > 0.0) {              // (a lucky breakdown, H_{j+1,j} = 0, leaves w)
      double* Wn = w.V + (size_t)(j + 1) * w.ld;
      const double inv = 1.0 / hn;
      const int hi = step_hi(v);
      for (int r = step_lo(v) + (int)threadIdx.x; r < hi; r += kGmThreads) {
        const double x = Wn[r] * inv;
        Wn[r] = x;
        if (prec) w.u[r] = v.dinv[r] * x;
      }
    }
    return;
  }
  if (threadIdx.x != 0) return;
  const double a = rotated;      // (step_sums ends with a barrier)
  const double b = hn;
  const double den = hypot(a, b);
  const double c = den > 0.0 ? a / den : 1.0, s = den > 0.0 ? b / den : 0.0;
  const double gj = st->g[j];
  st->cs[j] = c; st->sn[j] = s;
  Hj[j] = den; Hj[j + 1] = 0.0;
  const double gn = -s * gj;
  st->g[j + 1] = gn;
  st->g[j] = c * gj;
  st->gnorm = fabs(gn);
  st->iter += 1;
  st->j = j + 1;
  if (!(den > 0.0) || !(hn == hn)) { st->cyc_done = 1; if (!(den > 0.0)) st->status = ST_BREAKDOWN; return; }
  if (gn * gn <= st->thresh2 * st->bnorm2 || j + 1 >= st->m || st->iter >= st->max_iter || !(hn > 0.0)) {
    st->cyc_done = 1;
    return;
  }
  st->act[j + 1] = 1;
}

// End of a cycle: y = H^-1 g (back substitution over the k = j steps done)
// (one warp: lane c holds the right-hand sides c and c + 32, and the columns are
// eliminated from the last; one thread doing the rows took 59 us at k = 30)
__global__ void k_gm_solve_y(KrView v) {
  KrState* st = v.st;
  if (*((volatile int*)&st->status) != ST_RUNNING) return;
  const int k = st->j, l = threadIdx.x;
  double g0 = l < k ? st->g[l] : 0.0, g1 = l + 32 < k ? st->g[l + 32] : 0.0;
  for (int i = k - 1; i >= 0; --i) {
    const double* Hi = st->H + i * (kMaxRestart + 1);
    const double y = __shfl_sync(0xffffffffu, i < 32 ? g0 : g1, i & 31) / Hi[i];
    if (l == (i & 31)) st->y[i] = y;
    if (l < i) g0 = fma(-Hi[l], y, g0);
    if (l + 32 < i) g1 = fma(-Hi[l + 32], y, g1);
  }
}

// x += M^-1 (V y)
__global__ void k_gm_update_x(KrView v, GmVecs w) {
  KrState* st = v.st;
  if (*((volatile int*)&st->status) != ST_RUNNING) return;
  const int k = st->j;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < v.n; i += (long long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int c = 0; c < k; ++c) s += st->y[c] * w.V[(size_t)c * w.ld + i];
    w.x[i] += v.dinv[i] * s;
  }
}

// With a general (SSOR) preconditioner: t = V y (the correction before
// preconditioning), then x += M^-1 t.
__global__ void k_gm_vy(KrView v, GmVecs w, double* t) {
  KrState* st = v.st;
  if (*((volatile int*)&st->status) != ST_RUNNING) return;
  const int k = st->j;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < v.n; i += (long long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int c = 0; c < k; ++c) s += st->y[c] * w.V[(size_t)c * w.ld + i];
    t[i] = s;
  }
}
__global__ void k_gm_add_x(KrView v, double* x, const double* z) {
  if (*((volatile int*)&v.st->status) != ST_RUNNING) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < v.n; i += (long long)gridDim.x * blockDim.x)
    x[i] += z[i];
}

int grid1(long long n) { return (int)std::max(1LL, std::min<long long>((n + 255) / 256, 152LL * 8)); }

}  // namespace

#define NLGB_KR_T(LAUNCH)                                         \
  switch (A.tpr) {                                                \
    case 1: { constexpr int T = 1; LAUNCH; } break;               \
    case 2: { constexpr int T = 2; LAUNCH; } break;               \
    case 4: { constexpr int T = 4; LAUNCH; } break;               \
    case 8: { constexpr int T = 8; LAUNCH; } break;               \
    case 16: { constexpr int T = 16; LAUNCH; } break;             \
    default: { constexpr int T = 32; LAUNCH; } break;             \
  }

cudaError_t krylov_solve(const DeviceCRS& A, const double* dinv, const double* b, double* x,
                         int method, double eps, long long max_iter, int restart, cudaStream_t s,
                         KrylovResult* res, SsorPrecond* P) {
  const int n = A.n;
  const int tile_rows = A.tile_rows > 0 ? A.tile_rows : 128;
  const int n_tiles = std::max(1, (n + tile_rows - 1) / tile_rows);
  const int m = std::max(1, std::min(restart, kMaxRestart));
  // work vectors (+ two for GMRES's correction around a general preconditioner)
  const int n_vec = method == KRYLOV_BICGSTAB ? 7 : (m + 2 + (P ? 2 : 0));
  const size_t ld = (size_t)((n + 31) / 32 * 32);
  double* work = nullptr;
  double* part = nullptr;
  KrState* st = nullptr;
  NLGB_CUDA_TRY(cudaMallocAsync(&work, sizeof(double) * ld * n_vec + 256, s));
  cudaError_t e = cudaMallocAsync(&part, sizeof(double) * (size_t)n_tiles * kParts, s);
  if (e == cudaSuccess) e = cudaMallocAsync(&st, sizeof(KrState), s);
  double* mpart = nullptr;
  // step kernels (and BiCGSTAB's p and s): one CTA per SM (at least 256 rows each), two areas of
  // partials (a kernel reads one and writes the other)
  int dev = 0, sms = 152;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    sms = 152;
  }
  const int step_rows = std::max(256, (n + sms - 1) / sms);
  const int step_ctas = std::max(1, (n + step_rows - 1) / step_rows);
  const size_t part_area = (size_t)step_ctas * (m + 1);
  if (e == cudaSuccess && method == KRYLOV_GMRES) e = cudaMallocAsync(&mpart, sizeof(double) * 2 * part_area, s);
  KrState h;
  std::memset(&h, 0, sizeof(h));
  h.thresh2 = eps * eps;
  h.max_iter = max_iter;
  h.status = ST_RUNNING;
  h.m = m;
  if (e == cudaSuccess) e = cudaMemcpyAsync(st, &h, sizeof(h), cudaMemcpyHostToDevice, s);
  KrView v{n, tile_rows, n_tiles, A.rp, A.ci, A.va, dinv, part, st, mpart, m + 1, step_ctas, step_rows};
  long long launches = 0;
  auto poll = [&](int* status) {
    cudaError_t pe = cudaMemcpyAsync(status, &st->status, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (pe == cudaSuccess) pe = cudaStreamSynchronize(s);
    return pe;
  };
  if (e == cudaSuccess && method == KRYLOV_BICGSTAB) {
    BiVecs w{b, x, work, work + ld, work + 2 * ld, work + 3 * ld, work + 4 * ld, work + 5 * ld, work + 6 * ld};
    NLGB_KR_T((k_bi_init<T><<<n_tiles, kCTA, 0, s>>>(v, w)));
    k_bi_init_scalar<<<1, kCTA, 0, s>>>(v);
    launches += 2;
    const int threads = n <= kBiSmall * sms ? kCTA : kBiThreads, quarters = threads / kCTA;
    const int xr_ctas = std::min(threads == kCTA ? 2 * sms : sms, (n_tiles + quarters - 1) / quarters);
    int status = ST_RUNNING;
    long long it = 0;
    while (e == cudaSuccess && status == ST_RUNNING) {
      for (int c = 0; c < kChunk; ++c, ++it) {
        // (with a general preconditioner dinv is all ones: y = p, z = s,
        // then y = M^-1 p, z = M^-1 s)
        k_bi_p<<<step_ctas, threads, 0, s>>>(v, w, it, c > 0);
        if (P && e == cudaSuccess) e = P->apply(w.p, w.y, s);
        NLGB_KR_T((k_bi_v<T><<<n_tiles, kCTA, 0, s>>>(v, w)));
        k_bi_s<<<step_ctas, threads, 0, s>>>(v, w, it);
        if (P && e == cudaSuccess) e = P->apply(w.r, w.z, s);
        NLGB_KR_T((k_bi_t<T><<<n_tiles, kCTA, 0, s>>>(v, w)));
        k_bi_xr<<<xr_ctas, threads, 0, s>>>(v, w);
        launches += 5;
      }
      k_bi_end<<<1, kCTA, 0, s>>>(v, it - 1);
      launches += 1;
      if (e == cudaSuccess) e = cudaGetLastError();
      if (e == cudaSuccess) e = poll(&status);
    }
  } else if (e == cudaSuccess) {
    GmVecs w{b, x, work, work + (size_t)(m + 1) * ld, ld};
    double* t = P ? work + (size_t)(m + 2) * ld : nullptr;
    double* tz = P ? work + (size_t)(m + 3) * ld : nullptr;
    int status = ST_RUNNING;
    bool first = true;
    while (e == cudaSuccess && status == ST_RUNNING) {
      NLGB_KR_T((k_gm_residual<T><<<n_tiles, kCTA, 0, s>>>(v, w)));
      k_gm_start<<<1, kCTA, 0, s>>>(v, first ? 1 : 0);
      k_gm_scale0<<<grid1(n), 256, 0, s>>>(v, w, P ? 0 : 1);
      launches += 3;
      first = false;
      KrView v1 = v;               // the other area of partials
      v1.mpart = mpart + part_area;
      for (int j = 0; j < m; ++j) {
        if (P && e == cudaSuccess) e = P->apply(w.V + (size_t)j * ld, w.u, s);   // u = M^-1 V_j
        NLGB_KR_T((k_gm_spmv<T><<<step_ctas, kGmThreads, 0, s>>>(v, w, j)));
        k_gm_orth<<<step_ctas, kGmThreads, 0, s>>>(v1, w, j, 0, v.mpart);        // CGS2
        k_gm_orth<<<step_ctas, kGmThreads, 0, s>>>(v, w, j, 1, v1.mpart);
        k_gm_next<<<step_ctas + 1, kGmThreads, 0, s>>>(v, w, j, P ? 0 : 1);
        launches += 4;
      }
      k_gm_solve_y<<<1, 32, 0, s>>>(v);
      if (P) {
        k_gm_vy<<<grid1(n), 256, 0, s>>>(v, w, t);
        if (e == cudaSuccess) e = P->apply(t, tz, s);
        k_gm_add_x<<<grid1(n), 256, 0, s>>>(v, w.x, tz);
        launches += 1;
      } else {
        k_gm_update_x<<<grid1(n), 256, 0, s>>>(v, w);
      }
      launches += 2;
      if (e == cudaSuccess) e = cudaGetLastError();
      if (e == cudaSuccess) e = poll(&status);
    }
  }
  if (e == cudaSuccess) {
    NLGB_KR_T((k_kr_true<T><<<n_tiles, kCTA, 0, s>>>(v, b, x)));
    k_kr_true_scalar<<<1, kCTA, 0, s>>>(v);
    launches += 2;
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  count_launches(launches);
  cudaFreeAsync(work, s);
  if (part) cudaFreeAsync(part, s);
  if (st) cudaFreeAsync(st, s);
  if (mpart) cudaFreeAsync(mpart, s);
  if (e != cudaSuccess) return e;
  if (res) {
    res->status = h.status;
    res->iterations = h.iter;
    res->rel_residual = h.bnorm2 > 0 ? std::sqrt(h.rr / h.bnorm2) : 0.0;
    res->true_rel_residual = h.bnorm2 > 0 ? std::sqrt(h.rr_true / h.bnorm2) : 0.0;
  }
  return cudaSuccess;
}

}  // namespace nlgb
