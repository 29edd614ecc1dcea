// nlgb_persist.cuh -- the PCG iteration of one small or mid-size system as one
// persistent kernel (FP64, double-float, and the FP32 iteration of mixed
// precision).
//
// Replaces, like nlgb_solver.cu, the loop of OpenNL's
// nlSolveSystemIterative(NL_CG, Jacobi) (call sites:
// src/lib/OGF/scene_graph/NL/matrix.cpp:364,390-393).
//
// What bounds these sizes is latency: two scalar exchanges per iteration,
// and FP64 instructions, of which a warp issues one per 64 cycles on GB300
// (an SM one per 16, whatever the number of active lanes; measured with a
// dependent chain and with 4 to 32 warps).  A one-way message through L2
// costs about 885 cycles, a release/acquire one 1,710, an L2 hit 471.  Hence:
//   * a CTA keeps its rows' vectors in shared memory for the whole solve; an
//     exchanged word carries its iteration number in the same 16-byte access,
//     so that no fence is needed (and nothing in the loop invalidates L1);
//   * each thread keeps the nonzeros of its rows in registers (up to 10 per
//     lane and row, up to four rows), so that the SpMV's loop is LDS + FMA;
//   * x, r, p, q never go through L2.  A CTA holds a copy of p for the
//     columns of its rows that other CTAs own (the halo) and updates that
//     copy itself, p = z + beta p, from the z that the owner publishes
//     together with its r.z partials: p needs no exchange of its own;
//   * the rows of a CTA are dealt to its warps sorted by length, so that a
//     warp's rows have the same number of nonzeros (the 7-nonzero Laplacian
//     has rows of 5 to 9: 7 FP64 instructions per row instead of 9);
//   * block sums run in as few warp instructions as the tree has levels'
//     adds, spread over the four schedulers.
// Two forms.  Systems that kPersistCluster CTAs hold: one thread-block cluster, partial
// sums and z through distributed shared memory (a cluster barrier costs 378
// cycles), every CTA taking the scalar steps itself.  Above: a cooperative
// grid of one CTA per SM, one of which owns no rows, sums the partials and
// publishes alpha and beta (with every CTA polling every partial the polls
// themselves congested L2: 15,000 cycles per exchange on 512 tiles, 4,000
// with the reducing CTA).
// A tile's sums have the terms and the tree of the other executors, so the
// iterates are bit-identical to theirs.
//
// Measured, us per iteration, one cooperative kernel per iteration (mixed:
// three kernels and an IF node in a graph) -> this kernel: fairing 33 x 31
// FP64 10.7 -> 5.0, LSCM 72 x 57 12.1 -> 6.2, fairing 363 x 291 FP64
// 21.7 -> 11.3 and mixed 30 -> 11.4, LSCM 256 x 256 28.1 -> 15.1, fairing
// 650 x 650 (422,500 rows, three phase kernels before) 49.2 -> 29.0.  What is
// left at LSCM 256^2 (31,500 cycles): 9,300 in the SpMV, 4,900 in the x / r
// update and its sums, and 2 x 4,000 in the two exchanges through the
// reducing CTA.
#pragma once
#include "nlgb_persist.h"

namespace nlgb {
namespace {

// Codes a reducer publishes with a scalar.
enum : int { GO = 0, STOP = 1, STOP_AFTER_P = 2 };

__device__ __forceinline__ unsigned long long clock_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// One 16-byte slot: (payload, epoch), written and read as one access.
__device__ __forceinline__ void st_slot(ulonglong2* p, unsigned long long v, unsigned long long e) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
               :: "l"(p), "l"(v), "l"(e) : "memory");
}
__device__ __forceinline__ ulonglong2 ld_slot(const ulonglong2* p) {
  ulonglong2 r;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(r.x), "=l"(r.y) : "l"(p) : "memory");
  return r;
}
__device__ __forceinline__ unsigned long long bits_of(double v) { return (unsigned long long)__double_as_longlong(v); }
__device__ __forceinline__ unsigned long long bits_of(float v) { return (unsigned long long)__float_as_uint(v); }
__device__ __forceinline__ unsigned long long bits_of(float2 v) {
  return (unsigned long long)__float_as_uint(v.x) | ((unsigned long long)__float_as_uint(v.y) << 32);
}
__device__ __forceinline__ void from_bits(unsigned long long b, double& v) { v = __longlong_as_double((long long)b); }
__device__ __forceinline__ void from_bits(unsigned long long b, float& v) { v = __uint_as_float((unsigned)b); }
__device__ __forceinline__ void from_bits(unsigned long long b, float2& v) {
  v = make_float2(__uint_as_float((unsigned)b), __uint_as_float((unsigned)(b >> 32)));
}

__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" :: "r"(id), "r"(threads) : "memory");
}

// Distributed shared memory.
__device__ __forceinline__ unsigned peer_addr(const void* p, unsigned rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void st_peer(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" :: "r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void ld_peer(unsigned a, double& v) {
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_peer(unsigned a, float& v) {
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_peer(unsigned a, float2& v) {
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A bounded wait's bookkeeping: over() is true once the wait has to be given
// up (its own limit, or another CTA's error).
struct Wait {
  unsigned long long t0 = 0;
  unsigned int spins = 0;
  __device__ __forceinline__ bool over(const PersistArgs& a) {
    int* err = a.err;
    if ((++spins & 127u) != 0u) return false;
    const unsigned long long t = clock_ns();
    if (t0 == 0) t0 = t;
    if (*((volatile int*)err) != 0) return true;
    if (t - t0 > a.wait_ns) { atomicExch(err, 1); return true; }
    return false;
  }
};

// Sums of staged values in the order of block_sum: `nw` warps of M values
// each (value j of warp w at w * (M + 4) + j; the pad keeps the banks apart),
// per warp the butterfly's halving levels, then the warps in order.  A thread
// mapping of T lanes per row leaves only every T-th lane of a warp nonzero:
// M = 32 / T values, and the levels that would add zeros are gone.
//
// One warp's tree: lane 4w + c adds the values c, c + 4, ... of warp w.
// Returns warp w's total in the lanes of w.
template <int M>
__device__ __forceinline__ double warp_totals(const double* red, int nw) {
  const int l = threadIdx.x & 31, w = l >> 2, c = l & 3;
  constexpr int N = M >= 4 ? M / 4 : 1;
  double v[N];
#pragma unroll
  for (int j = 0; j < N; ++j) v[j] = (w < nw && c + 4 * j < M) ? red[w * (M + 4) + c + 4 * j] : 0.0;
#pragma unroll
  for (int h = N / 2; h > 0; h >>= 1)
#pragma unroll
    for (int j = 0; j < h; ++j) v[j] += v[j + h];
  double s = v[0];
  if constexpr (M >= 4) s += __shfl_xor_sync(0xffffffffu, s, 2);
  if constexpr (M >= 2) s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}
// The totals of warps w0 .. w0 + nw - 1 in order (w0 may differ between
// lanes; rolled: see serial_sum).
__device__ __forceinline__ double in_order(double s, int w0, int nw) {
  double tot = __shfl_sync(0xffffffffu, s, 4 * w0);
#pragma unroll 1
  for (int i = 1; i < nw; ++i) tot += __shfl_sync(0xffffffffu, s, 4 * (w0 + i));
  return tot;
}
// The butterfly of one warp's 32 values by 16 lanes: lane i adds the values i
// and i + 16, then the lanes' levels 8, 4, 2, 1.
__device__ __forceinline__ double half_levels(double a, double b) {
  double s = a + b;
  s += __shfl_xor_sync(0xffffffffu, s, 8);
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}

template <int MODE> struct Traits;
template <> struct Traits<kPersistDouble> { using V = double; using V2 = double2; };
template <> struct Traits<kPersistDf> { using V = float2; using V2 = float4; };
template <> struct Traits<kPersistMixed> { using V = float; using V2 = float2; };

// The double-float block sum (df_block_sum's order).
__device__ __forceinline__ float2 df_warp_sum(float2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float2 t;
    t.x = __shfl_xor_sync(0xffffffffu, v.x, o);
    t.y = __shfl_xor_sync(0xffffffffu, v.y, o);
    v = df::dadd(v, t);
  }
  return v;
}

// One lane's running row sum (row_dot's / row_dot_df's terms and order).
template <int MODE>
struct RowSum {
  typename Traits<MODE>::V s;
  __device__ __forceinline__ void clear() {
    if constexpr (MODE == kPersistDf) s = make_float2(0.f, 0.f);
    else s = 0;
  }
  __device__ __forceinline__ void add(typename Traits<MODE>::V a, typename Traits<MODE>::V x) {
    if constexpr (MODE == kPersistDf) {   // s = (head, tail), not normalised
      const float pr = df::mul(a.x, x.x);
      float e = df::fma(a.x, x.x, -pr);
      e = df::fma(a.x, x.y, e);
      e = df::fma(a.y, x.x, e);
      const float2 t = df::two_sum(s.x, pr);
      s.x = t.x;
      s.y = df::add(s.y, df::add(t.y, e));
    } else {
      s = fma(a, x, s);
    }
  }
  template <int T>
  __device__ __forceinline__ typename Traits<MODE>::V total() const {
    if constexpr (MODE == kPersistDf) {
      float2 v = df::fast_two_sum(s.x, s.y);
#pragma unroll
      for (int o = T / 2; o > 0; o >>= 1) {
        float2 t;
        t.x = __shfl_xor_sync(0xffffffffu, v.x, o);
        t.y = __shfl_xor_sync(0xffffffffu, v.y, o);
        v = df::dadd(v, t);
      }
      return v;
    } else {
      return subwarp_sum<T, typename Traits<MODE>::V>(s);
    }
  }
};
template <int MODE>
__device__ __forceinline__ typename Traits<MODE>::V ld_value(const SysView& s, int k) {
  if constexpr (MODE == kPersistMixed) return __ldg(s.va32 + k);
  else if constexpr (MODE == kPersistDf) return __ldg(s.vadf + k);
  else return __ldg(s.va + k);
}

// The scalar steps of a running iteration, on one thread's registers: the
// results and decisions of scalar_after_pq / scalar_after_xr /
// scalar_after_mx_cr while the iteration goes on (comparisons of
// non-negative doubles as integers: an FP64 comparison costs 64 cycles like
// any FP64 instruction, and the thresholds do not change).  Anything else --
// convergence, a limit, a breakdown -- is left to those functions.
template <int MODE>
struct Scalars {
  double rho, alpha, beta;
  unsigned long long thr;      // stop at r.r <= thr
  long long left;              // iterations before a limit
  __device__ __forceinline__ void load(const SysState& st) {
    rho = st.rho; alpha = st.alpha; beta = st.beta;
    double t = (MODE == kPersistMixed ? st.thresh2 : st.rthresh2) * st.bnorm2;
    left = st.max_iter - st.iter;
    if constexpr (MODE == kPersistMixed) {
      t = fmax(t, st.in_thresh2 * st.in_rr0);
      left = min(left, (long long)(st.in_max - st.in_iter));
    }
    thr = (unsigned long long)__double_as_longlong(t);
  }
  static __device__ __forceinline__ bool pos(double v) {   // finite_pos: 0 < v < 1e300
    return (unsigned long long)__double_as_longlong(v) - 1ULL <
           (unsigned long long)__double_as_longlong(1.0e300) - 1ULL;
  }
  __device__ __forceinline__ bool after_pq(double pq) {
    alpha = rho / pq;
    return pos(pq);
  }
  // true: the iteration goes on (n iterations of this launch done before it)
  __device__ __forceinline__ bool after_xr(double rz, double rr, long long n) const {
    const unsigned long long b = (unsigned long long)__double_as_longlong(rr);
    return pos(rz) && b > thr && b <= (unsigned long long)__double_as_longlong(1.0e300) && n + 1 < left;
  }
  __device__ __forceinline__ void advance(double rz) { beta = rz / rho; rho = rz; }
  // the state after n iterations that went on
  __device__ __forceinline__ void store(SysState& st, long long n) const {
    st.rho = rho; st.alpha = alpha; st.beta = beta;
    st.iter += n;
    if constexpr (MODE == kPersistMixed) st.in_iter += (int)n;
  }
};

// nw values in order.  Rolled on purpose: what runs once per iteration in one
// warp is bound by instruction fetch (the unrolled form took 2,500 cycles for
// three values, this one 600).
__device__ __forceinline__ double serial_sum(const double* v, int nw) {
  double s = v[0];
#pragma unroll 1
  for (int i = 1; i < nw; ++i) s += v[i];
  return s;
}

// Iterations of this launch at most: a chunk of a mixed system takes a launch
// per reliable update, and ends where its budget does.
__device__ __forceinline__ long long launch_iters(const PersistArgs& a, const SysState& st) {
  return st.iter_stop > 0 ? min(a.iters, st.iter_stop - st.iter) : a.iters;
}

// Tells the host that this launch is over (one thread; the state itself is for
// the kernels that the host queues then).
template <int MODE>
__device__ __forceinline__ void tell_done(const PersistArgs& a, const SysState& st) {
  if (a.done == nullptr) return;
  const unsigned end = st.status != ST_RUNNING                  ? kPersistStopped
                       : MODE == kPersistMixed && st.mode == 0 ? kPersistUpdate
                                                               : kPersistPaused;
  *reinterpret_cast<volatile unsigned int*>(a.done) = a.done_value + end;
}

// ---------------------------------------------------------------------------
// The reducing CTA of the grid form (256 threads): sums the tiles' partials
// as they arrive, takes the scalar steps and publishes alpha and beta.
// Sixteen half-warps: half-warp h sums the tiles of canonical warp h mod 8
// of value h / 8 (canon_reduce's order: thread t adds tiles t, t + 256, ...;
// then each warp's butterfly; then the warps in order).
// ---------------------------------------------------------------------------
template <int MODE>
__device__ void reducer(const PersistArgs& a, SysState& sst) {
  __shared__ double tot[2][8];
  __shared__ int failed, stop;
  const SysView& s = a.s;
  const int tid = threadIdx.x;
  if (tid >= kCTA) return;
  const int i = tid & 15, cw = (tid >> 4) & 7, hv = tid >> 7;   // lane of the half-warp, canonical warp, value
  const int nw = min(kWarps, (s.n_tiles + 31) / 32);
  Scalars<MODE> sc;
  sc.load(sst);
  const unsigned long long base = (unsigned long long)sst.coop_epoch;
  const long long iters = launch_iters(a, sst);
  long long it = 0;
  int abort_now = 0;
  if (tid == 0) { failed = 0; stop = 0; }
  bar_sync(1, kCTA);

  // Half-warp sums of the tiles of canonical warp cw: lane i takes the tiles of
  // canonical lanes i and i + 16 (rolled: see serial_sum).
  auto gather = [&](const ulonglong2* slots, unsigned long long e) {
    double sa = 0.0, sb = 0.0;
    if (cw < nw) {
      Wait w;
#pragma unroll 1
      for (int t = cw * 32 + i; t < s.n_tiles; t += kCTA) {
        const bool two = t + 16 < s.n_tiles;
        ulonglong2 va, vb;
        do {
          va = ld_slot(slots + t);
          vb = ld_slot(slots + (two ? t + 16 : t));
        } while ((va.y != e || vb.y != e) && !w.over(a));
        if (va.y != e || vb.y != e) { failed = 1; break; }
        double v;
        from_bits(va.x, v);
        sa = t < kCTA ? v : sa + v;
        from_bits(vb.x, v);
        if (two) sb = t < kCTA ? v : sb + v;
      }
    }
    __syncwarp();
    return half_levels(sa, sb);
  };

  for (;;) {
    const unsigned long long e = base + (unsigned long long)it + 1ULL;
    // the abort flag (host memory) is read every fourth iteration of the solve (a
    // launch of a mixed system may end after fewer)
    if (tid == 0 && s.abort_flag != nullptr && ((base + it) & 3) == 3) abort_now = *s.abort_flag;
    if (hv == 0) {
      const double v = gather(a.slot, e);
      if (i == 0) tot[0][cw] = v;
    }
    bar_sync(1, kCTA);
    if (tid == 0) {
      const double pq = serial_sum(tot[0], nw);
      const bool go = sc.after_pq(pq) && !failed;
      st_slot(a.ctl, bits_of(sc.alpha), (e << 8) | (unsigned)(go ? GO : STOP));
      if (!go) {
        sc.store(sst, it);
        if (failed) sst.status = ST_DEVICE_ERR;
        else scalar_after_pq(&sst, pq);
      }
      stop = go ? 0 : 1;
    }
    bar_sync(1, kCTA);
    if (stop) break;
    const double v = gather(a.slot + (size_t)(1 + hv) * s.n_tiles, e);
    if (i == 0) tot[hv][cw] = v;
    bar_sync(1, kCTA);
    if (tid < 32) {
      const int k = tid & 1;
      const double sum = serial_sum(tot[k], nw);
      const double rr = __shfl_sync(0xffffffffu, sum, 1);
      if (tid == 0) {
        if (sc.after_xr(sum, rr, it) && it + 1 < iters && !abort_now && !failed) {
          sc.advance(sum);
          st_slot(a.ctl + 8, bits_of(sc.beta), (e << 8) | (unsigned)GO);
        } else {
          sc.store(sst, it);
          if (failed) sst.status = ST_DEVICE_ERR;
          else if constexpr (MODE == kPersistMixed) scalar_after_mx_cr(&sst, sum, rr);
          else scalar_after_xr(&sst, sum, rr);
          if (sst.status == ST_RUNNING && abort_now) sst.status = ST_ABORTED;
          // still running: this launch's iterations are used up
          const int code = sst.status != ST_RUNNING || MODE == kPersistMixed ? STOP : STOP_AFTER_P;
          st_slot(a.ctl + 8, bits_of(sst.beta), (e << 8) | (unsigned)code);
          stop = 1;
        }
      }
    }
    ++it;
    bar_sync(1, kCTA);
    if (stop) break;
  }
  if (tid == 0) {
    sst.coop_epoch += it;
    sst.guard += (it + 3) / 4;
    *s.st = sst;
    tell_done<MODE>(a, sst);
  }
}

// NC: rows per lane group whose nonzeros stay in registers.
template <int T, int MODE, bool CLUSTER, int NC>
__global__ void __launch_bounds__(kPersistBlock, 1) k_persist(PersistArgs a) {
  using V = typename Traits<MODE>::V;
  using V2 = typename Traits<MODE>::V2;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SysState sst;
  __shared__ double s_scalar[2];            // alpha, beta
  __shared__ int s_code[2], s_failed, s_abort;
  __shared__ double s_part[CLUSTER ? 3 : 1][CLUSTER ? kPersistClusterTiles : 1];   // cluster form: every tile's partials
  __shared__ double s_tot[2][8];
  __shared__ float2 s_dft[MODE == kPersistDf ? kPersistSlots * 2 : 1][8];
  const SysView& s = a.s;
  const int C = a.lay.ctas, cta = (int)blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = (int)blockDim.x >> 5;
  const int R = s.tile_rows;

  if (threadIdx.x == 0) { sst = *s.st; s_code[0] = s_code[1] = GO; s_failed = 0; s_abort = 0; }
  __syncthreads();
  const long long iters = launch_iters(a, sst);
  if (sst.status != ST_RUNNING || (MODE == kPersistMixed && sst.mode != 1) || iters <= 0) {
    if (cta == 0 && threadIdx.x == 0) tell_done<MODE>(a, sst);
    return;
  }
  if constexpr (!CLUSTER) {
    if (cta == C) { reducer<MODE>(a, sst); return; }
  }

  // This CTA's tiles: a contiguous range, the first `extra` CTAs one more.
  const int per = s.n_tiles / C, extra = s.n_tiles % C;
  const int t0 = cta * per + min(cta, extra);
  const int cnt = per + (cta < extra ? 1 : 0);
  const int row0 = t0 * R, rows = min(s.n, (t0 + cnt) * R) - row0;
  const int cap = a.lay.slots * R;
  const int H = a.lay.halo_n[cta];
  const int* halo = a.lay.halo + (size_t)cta * a.lay.halo_stride;

  // Shared memory: p of the own rows and of the halo, z of the halo, then q,
  // z, r, x, 1/diag of the own rows, and two staged values per tile.
  V* ps = reinterpret_cast<V*>(smem);
  V* hz = ps + cap + a.lay.halo_cap;
  V* qs = hz + a.lay.halo_cap;
  V* zs = qs + cap;
  V* rs = zs + cap;
  V* xs = rs + cap;
  V* ds = xs + cap;
  double* red = reinterpret_cast<double*>(ds + cap);

  V *wx, *wr, *wp;
  const V* gd;
  if constexpr (MODE == kPersistMixed) {
    wx = s.c32; wr = s.r32; wp = s.p32;
    gd = s.dinv32;
  } else if constexpr (MODE == kPersistDf) {
    wx = reinterpret_cast<float2*>(s.x); wr = reinterpret_cast<float2*>(s.r); wp = reinterpret_cast<float2*>(s.p);
    gd = s.dinvdf;
  } else {
    wx = s.x; wr = s.r; wp = s.p;
    gd = s.dinv;
  }
  for (int i = threadIdx.x; i < rows; i += blockDim.x) {
    xs[i] = __ldcg(wx + row0 + i);
    const V r = __ldcg(wr + row0 + i), d = __ldg(gd + row0 + i);
    rs[i] = r;
    ds[i] = d;
    V p = __ldcg(wp + row0 + i);
    // (mixed: the p update comes first; p = beta p + D^-1 r)
    if constexpr (MODE == kPersistMixed) p = fmaf(float(sst.beta), p, d * r);
    ps[i] = p;
  }
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    int c = halo[i];
    if constexpr (CLUSTER) {
      const int rk = c >> 16;
      c = (rk * per + min(rk, extra)) * R + (c & 0xffff);
    }
    V p = __ldcg(wp + c);
    if constexpr (MODE == kPersistMixed) p = fmaf(float(sst.beta), p, __ldg(gd + c) * __ldcg(wr + c));
    ps[cap + i] = p;
  }

  // nonzeros per lane and row in registers: the first rows are the longest
  constexpr int U = NC <= 2 ? 10 : 12, U1 = NC <= 2 ? 10 : 8;
  constexpr int RPW = 32 / T;                    // rows per warp
  constexpr int RPP = kCTA / T;                  // chains of a tile: rows j, j + RPP, ...
  constexpr int M = 32 / T;                      // chains per canonical warp
  const bool one_pass = R <= RPP;                // a chain is one row
  const int nch = (rows + RPW - 1) / RPW;
  const int nw_pq = (min(R, RPP) + M - 1) / M;   // canonical warps with chains
  const int nw_xr = ((R + 1) / 2 + 31) / 32;     // canonical warps with row pairs
  const int xr_sl = warp / nw_xr;                // tile slot of this warp's first row pairs
  const unsigned long long base = (unsigned long long)sst.coop_epoch;
  // The staged value of chain j of tile slot sl.
  auto chain_at = [&](int sl, int j) { return sl * 2 * kPersistRed + (j / M) * (M + 4) + (j % M); };

  // The rows this lane group keeps in registers.
  V av[NC][U];
  unsigned cv[NC][U / 2];
  // row (0xffff: none) | own length << 16 | the warp's longest << 21 | more than U << 26
  unsigned meta[NC];
  int pos_r[NC];
#pragma unroll
  for (int ch = 0; ch < NC; ++ch) {
    // (the longest rows first; every other round backwards, so that no warp gets the longest of each)
    const int idx = (ch * nwarps + ((ch & 1) ? nwarps - 1 - warp : warp)) * RPW + lane / T;
    unsigned row = 0xffffu, len = 0, more = 0;
    pos_r[ch] = 0;
#pragma unroll
    for (int u = 0; u < U / 2; ++u) cv[ch][u] = 0u;
    if (idx < rows) {
      const int r = a.lay.perm[row0 + idx];
      const int k0 = s.rp[row0 + r] + lane % T, k1 = s.rp[row0 + r + 1];
      row = (unsigned)r;
      pos_r[ch] = chain_at(r / R, r % R);
      more = k0 + (ch == 0 ? U : U1) * T < k1 ? 1u : 0u;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if ((ch == 0 || u < U1) && k0 + u * T < k1) {
          av[ch][u] = ld_value<MODE>(s, k0 + u * T);
          cv[ch][u >> 1] |= (unsigned)a.lay.lci[k0 + u * T] << (16 * (u & 1));
          len = u + 1;
        }
    }
    meta[ch] = row | len << 16 | __reduce_max_sync(0xffffffffu, len) << 21 | more << 26;
  }
  long long it = 0;
  int abort_now = 0;
  Scalars<MODE> sc;
  if constexpr (CLUSTER) sc.load(sst);
  if constexpr (CLUSTER) cluster_barrier();   // every CTA's shared memory is set up
  else __syncthreads();

  // Publish a tile's value k (called by all lanes of one warp).
  auto publish = [&](int k, int tile, double v, unsigned long long e) {
    if constexpr (CLUSTER) {
      if (lane < C) st_peer(peer_addr(&s_part[k][tile], (unsigned)lane), v);
    } else {
      if (lane == 0) st_slot(a.slot + (size_t)k * s.n_tiles + tile, bits_of(v), e);
    }
  };
  // Grid form: thread 0 waits for scalar `which` of epoch e.
  auto wait_scalar = [&](int which, unsigned long long e) {
    if (threadIdx.x == 0) {
      const ulonglong2* slot = a.ctl + 8 * which;
      Wait w;
      ulonglong2 v = ld_slot(slot);
      while ((v.y >> 8) != e) {
        if (w.over(a)) { s_failed = 1; break; }
        v = ld_slot(slot);
      }
      from_bits(v.x, s_scalar[which]);
      s_code[which] = (int)(v.y & 0xffULL);
    }
    __syncthreads();
  };
  // Cluster form: the canonical sum of value k from the tiles' partials (at
  // most two canonical warps of tiles).
  auto cluster_sum = [&](int k) {
    const int i = lane & 15, t = (lane >> 4) * 32 + i;
    const double va = t < s.n_tiles ? s_part[k][t] : 0.0;
    const double vb = t + 16 < s.n_tiles ? s_part[k][t + 16] : 0.0;
    const double h = half_levels(va, vb);
    double tot = __shfl_sync(0xffffffffu, h, 0);
    if (s.n_tiles > 32) tot += __shfl_sync(0xffffffffu, h, 16);
    return tot;
  };
  // Double-float: the canonical warps' sums of staged values (two syncs).
  auto df_trees = [&](int K, int nw, int m, int k0, unsigned long long e) {
    if constexpr (MODE == kPersistDf) {
      for (int u = warp; u < cnt * K * 8; u += nwarps) {
        const int sk = u >> 3, cw = u & 7;
        const float2* r = reinterpret_cast<const float2*>(red + ((sk / K) * 2 + sk % K) * kPersistRed) + cw * (m + 4);
        // lane i of the canonical warp holds chain i / (32 / m) (others zero)
        const int st = 32 / m;
        float2 v = make_float2(0.f, 0.f);
        if (cw < nw && lane % st == 0) v = r[lane / st];
        v = df_warp_sum(v);
        if (lane == 0) s_dft[sk][cw] = v;
      }
      __syncthreads();
      for (int sk = warp; sk < cnt * K; sk += nwarps) {
        float2 t = s_dft[sk][0];
#pragma unroll
        for (int i = 1; i < 8; ++i) t = df::dadd(t, s_dft[sk][i]);
        publish(k0 + sk % K, t0 + sk / K, df::to_double(t), e);
      }
    }
  };

  for (;;) {
    const unsigned long long e = base + (unsigned long long)it + 1ULL;
    if constexpr (CLUSTER) {
      // the abort flag (host memory) is read every fourth iteration of the solve by
      // CTA 0, which hands it to the others before the iteration's second barrier
      if (cta == 0 && threadIdx.x == 0 && s.abort_flag != nullptr && ((base + it) & 3) == 3) abort_now = *s.abort_flag;
    }
    // q = A p; where a chain is one row, its p.q product too
    auto finish_row = [&](int row, int pos, V q) {
      qs[row] = q;
      if (one_pass) {
        if constexpr (MODE == kPersistDf)
          reinterpret_cast<float2*>(red)[pos] = df::mac(make_float2(0.f, 0.f), ps[row], q);
        else if constexpr (MODE == kPersistMixed) red[pos] = to_double_int(ps[row] * q);
        else red[pos] = fma(ps[row], q, 0.0);
      }
    };
    RowSum<MODE> sum[NC];
#pragma unroll
    for (int ch = 0; ch < NC; ++ch) {
      sum[ch].clear();
      V xv[U];
      const int len = (int)(meta[ch] >> 16) & 31, longest = (int)(meta[ch] >> 21) & 31;
#pragma unroll
      for (int u = 0; u < (ch == 0 ? U : U1); ++u) {
        if (u >= longest) break;
        xv[u] = ps[(cv[ch][u >> 1] >> (16 * (u & 1))) & 0xffffu];
      }
#pragma unroll
      for (int u = 0; u < (ch == 0 ? U : U1); ++u) {
        if (u >= longest) break;
        if (u < len) sum[ch].add(av[ch][u], xv[u]);
      }
      if (meta[ch] >> 26) {
        const int* rp = s.rp + row0 + (meta[ch] & 0xffffu);
#pragma unroll 1
        for (int k = __ldg(rp) + lane % T + (ch == 0 ? U : U1) * T; k < __ldg(rp + 1); k += T)
          sum[ch].add(ld_value<MODE>(s, k), ps[__ldg(a.lay.lci + k)]);
      }
      __syncwarp();
    }
    if constexpr (T == 2 && NC % 2 == 0 && MODE == kPersistDouble) {
      // two rows' lane pairs share one addition: the first lane finishes row
      // ch, the second row ch + 1 (addition commutes: the butterfly's bits)
#pragma unroll
      for (int ch = 0; ch < NC; ch += 2) {
        const bool second = (lane & 1) != 0;
        const double keep = second ? sum[ch + 1].s : sum[ch].s;
        const double q = keep + __shfl_xor_sync(0xffffffffu, second ? sum[ch].s : sum[ch + 1].s, 1);
        const int row = (int)((second ? meta[ch + 1] : meta[ch]) & 0xffffu);
        if (row != 0xffff) finish_row(row, second ? pos_r[ch + 1] : pos_r[ch], q);
      }
    } else {
#pragma unroll
      for (int ch = 0; ch < NC; ++ch) {
        const V q = sum[ch].template total<T>();
        const int row = (int)(meta[ch] & 0xffffu);
        if (row != 0xffff && lane % T == 0) finish_row(row, pos_r[ch], q);
      }
    }
#pragma unroll 1
    for (int ch = NC * nwarps + warp; ch < nch; ch += nwarps) {   // rows beyond the registers
      const int idx = ch * RPW + lane / T;
      int row = -1, k0 = 0, k1 = 0;
      if (idx < rows) {
        row = __ldg(a.lay.perm + row0 + idx);
        k0 = __ldg(s.rp + row0 + row);
        k1 = __ldg(s.rp + row0 + row + 1);
      }
      RowSum<MODE> rsum;
      rsum.clear();
#pragma unroll 2
      for (int k = k0 + lane % T; k < k1; k += T) rsum.add(ld_value<MODE>(s, k), ps[__ldg(a.lay.lci + k)]);
      __syncwarp();
      const V q = rsum.template total<T>();
      if (row >= 0 && lane % T == 0) finish_row(row, chain_at(row / R, row % R), q);
    }
    if (one_pass)   // chains of a short last tile
#pragma unroll 1
      for (int i = rows + (int)threadIdx.x; i < cnt * R; i += blockDim.x) red[chain_at(i / R, i % R)] = 0.0;
    __syncthreads();
    if (!one_pass) {
      // chain j of a tile: its rows in order
#pragma unroll 1
      for (int u = threadIdx.x; u < cnt * RPP; u += blockDim.x) {
        const int sl = u / RPP, j = u % RPP, hi = min(rows, (sl + 1) * R);
        if constexpr (MODE == kPersistDf) {
          float2 acc = make_float2(0.f, 0.f);
#pragma unroll 1
          for (int r = sl * R + j; r < hi; r += RPP) acc = df::mac(acc, ps[r], qs[r]);
          reinterpret_cast<float2*>(red)[chain_at(sl, j)] = acc;
        } else {
          double acc = 0.0;
#pragma unroll 1
          for (int r = sl * R + j; r < hi; r += RPP) {
            if constexpr (MODE == kPersistMixed) acc += to_double_int(ps[r] * qs[r]);
            else acc = fma(ps[r], qs[r], acc);
          }
          red[chain_at(sl, j)] = acc;
        }
      }
      __syncthreads();
    }
    if constexpr (MODE == kPersistDf) {
      df_trees(1, nw_pq, M, 0, e);
    } else if (T == 1 && cnt == 1) {
      // one tile: the butterflies over the half-warps of four warps
      if (warp < 4) {
        const int cw = threadIdx.x >> 4, i = lane & 15;
        const double* r = red + cw * 36 + i;
        const double h = half_levels(cw < nw_pq ? r[0] : 0.0, cw < nw_pq ? r[16] : 0.0);
        if (i == 0) s_tot[0][cw] = h;
        bar_sync(2, 128);
        if (warp == 0) publish(0, t0, serial_sum(s_tot[0], nw_pq), e);
      }
    } else {
#pragma unroll 1
      for (int sl = warp; sl < cnt; sl += nwarps)
        publish(0, t0 + sl, in_order(warp_totals<M>(red + sl * 2 * kPersistRed, nw_pq), 0, nw_pq), e);
    }
    if constexpr (CLUSTER) {
      cluster_barrier();
      if (warp == 0) {
        const double pq = cluster_sum(0);
        if (lane == 0) {
          if (!sc.after_pq(pq)) {
            sc.store(sst, it);
            scalar_after_pq(&sst, pq);
            s_code[0] = STOP;
          }
          s_scalar[0] = sc.alpha;
        }
      }
      __syncthreads();
    } else {
      wait_scalar(0, e);
      if (s_failed) break;
    }
    if (s_code[0] != GO) break;
    // r -= alpha q, z = D^-1 r, r.z, r.r: canonical warp w of tile slot sl
    // handles the row pairs 32 w + lane of the tile
    const double alpha = s_scalar[0];
#pragma unroll 1
    for (int u = warp, sl = xr_sl; u < cnt * nw_xr; u += nwarps, sl = u / nw_xr) {
      const int w = u - sl * nw_xr;
      const int lo = sl * R, hi = min(rows, lo + R), i = lo + 2 * (32 * w + lane);
      ulonglong2* zo = a.zslot + row0;
      const bool pair = i + 1 < hi;
      const bool tail = w == 0 && lane == 0 && ((hi - lo) & 1) != 0;   // an odd last row: thread 0, after its pair
      if constexpr (MODE == kPersistDf) {
        const float2 na = df::neg(df::from_double(alpha));
        float2 v0 = make_float2(0.f, 0.f), v1 = make_float2(0.f, 0.f);
        if (pair) {
          const float4 rv = *reinterpret_cast<const float4*>(rs + i), qv = *reinterpret_cast<const float4*>(qs + i);
          const float4 dv = *reinterpret_cast<const float4*>(ds + i);
          const float2 ra = df::mac(df::make(rv.x, rv.y), na, df::make(qv.x, qv.y));
          const float2 rb = df::mac(df::make(rv.z, rv.w), na, df::make(qv.z, qv.w));
          const float2 za = df::dmul(df::make(dv.x, dv.y), ra), zb = df::dmul(df::make(dv.z, dv.w), rb);
          v0 = df::mac(v0, za, ra); v0 = df::mac(v0, zb, rb);
          v1 = df::mac(v1, ra, ra); v1 = df::mac(v1, rb, rb);
          *reinterpret_cast<float4*>(rs + i) = make_float4(ra.x, ra.y, rb.x, rb.y);
          *reinterpret_cast<float4*>(zs + i) = make_float4(za.x, za.y, zb.x, zb.y);
          if constexpr (!CLUSTER) { st_slot(zo + i, bits_of(za), e); st_slot(zo + i + 1, bits_of(zb), e); }
        }
        if (tail) {
          const int j = hi - 1;
          const float2 r = df::mac(rs[j], na, qs[j]), z = df::dmul(ds[j], r);
          v0 = df::mac(v0, z, r);
          v1 = df::mac(v1, r, r);
          rs[j] = r;
          zs[j] = z;
          if constexpr (!CLUSTER) st_slot(zo + j, bits_of(z), e);
        }
        float2* st = reinterpret_cast<float2*>(red + sl * 2 * kPersistRed) + w * 36 + lane;
        st[0] = v0;
        st[kPersistRed] = v1;
      } else {
        double rz = 0.0, rr = 0.0;
        if (pair) {
          V2 rv = *reinterpret_cast<const V2*>(rs + i), zv;
          const V2 qv = *reinterpret_cast<const V2*>(qs + i), dv = *reinterpret_cast<const V2*>(ds + i);
          if constexpr (MODE == kPersistMixed) {
            const float al = float(alpha);
            rv.x = fmaf(-al, qv.x, rv.x); rv.y = fmaf(-al, qv.y, rv.y);
            zv.x = dv.x * rv.x; zv.y = dv.y * rv.y;
            rz = to_double_int(fmaf(zv.y, rv.y, zv.x * rv.x));
            rr = to_double_int(fmaf(rv.y, rv.y, rv.x * rv.x));
          } else {
            rv.x = fma(-alpha, qv.x, rv.x); rv.y = fma(-alpha, qv.y, rv.y);
            zv.x = dv.x * rv.x; zv.y = dv.y * rv.y;
            rz = fma(zv.x, rv.x, rz); rz = fma(zv.y, rv.y, rz);
            rr = fma(rv.x, rv.x, rr); rr = fma(rv.y, rv.y, rr);
          }
          *reinterpret_cast<V2*>(rs + i) = rv;
          *reinterpret_cast<V2*>(zs + i) = zv;
          if constexpr (!CLUSTER) { st_slot(zo + i, bits_of(zv.x), e); st_slot(zo + i + 1, bits_of(zv.y), e); }
        }
        if (tail) {
          const int j = hi - 1;
          V ri, zi;
          if constexpr (MODE == kPersistMixed) {
            ri = fmaf(-float(alpha), qs[j], rs[j]);
            zi = ds[j] * ri;
            rz += double(zi * ri);
            rr += double(ri * ri);
          } else {
            ri = fma(-alpha, qs[j], rs[j]);
            zi = ds[j] * ri;
            rz = fma(zi, ri, rz);
            rr = fma(ri, ri, rr);
          }
          rs[j] = ri;
          zs[j] = zi;
          if constexpr (!CLUSTER) st_slot(zo + j, bits_of(zi), e);
        }
        // up to four canonical warps: both values side by side (one tree)
        double* st = red + sl * 2 * kPersistRed + w * 36 + lane;
        st[0] = rz;
        st[nw_xr <= 4 ? nw_xr * 36 : kPersistRed] = rr;
      }
    }
    __syncthreads();
    if constexpr (MODE == kPersistDf) {
      df_trees(2, nw_xr, 32, 1, e);
    } else if (cnt == 1 && nw_xr <= 4) {
      // half-warp h: canonical warp h mod nw of value h / nw (staged in a row)
      if (warp < 4) {
        const int h = threadIdx.x >> 4, i = lane & 15;
        const bool on = h < 2 * nw_xr;
        const double* r = red + h * 36 + i;
        const double v = half_levels(on ? r[0] : 0.0, on ? r[16] : 0.0);
        if (on && i == 0) s_tot[h >= nw_xr ? 1 : 0][h >= nw_xr ? h - nw_xr : h] = v;
        bar_sync(2, 128);
        if (warp < 2) publish(1 + warp, t0, serial_sum(s_tot[warp], nw_xr), e);
      }
    } else if (nw_xr <= 4) {
#pragma unroll 1
      for (int sl = warp; sl < cnt; sl += nwarps) {
        // lanes 0-15 finish r.z, lanes 16-31 r.r
        const double v = in_order(warp_totals<32>(red + sl * 2 * kPersistRed, 2 * nw_xr), (lane >> 4) * nw_xr, nw_xr);
        publish(1, t0 + sl, __shfl_sync(0xffffffffu, v, 0), e);
        publish(2, t0 + sl, __shfl_sync(0xffffffffu, v, 16), e);
      }
    } else {
#pragma unroll 1
      for (int u = warp; u < 2 * cnt; u += nwarps)
        publish(1 + (u & 1), t0 + (u >> 1),
                in_order(warp_totals<32>(red + u * kPersistRed, nw_xr), 0, nw_xr), e);
    }
    // x += alpha p (off the critical path)
#pragma unroll 1
    for (int i = threadIdx.x; i < rows; i += blockDim.x) {
      if constexpr (MODE == kPersistMixed) xs[i] = fmaf(float(alpha), ps[i], xs[i]);
      else if constexpr (MODE == kPersistDf) xs[i] = df::mac(xs[i], df::from_double(alpha), ps[i]);
      else xs[i] = fma(alpha, ps[i], xs[i]);
    }
    ++it;
    if constexpr (CLUSTER) {
      if (cta == 0 && threadIdx.x == 0 && abort_now) {
#pragma unroll 1
        for (int c = 0; c < C; ++c) {
          const unsigned pa = peer_addr(&s_abort, (unsigned)c);
          asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(pa), "r"(1) : "memory");
        }
      }
      cluster_barrier();
      if (warp < 2) {
        const double v = cluster_sum(1 + warp);
        if (lane == 0) s_tot[warp][0] = v;
        bar_sync(2, 64);
        if (threadIdx.x == 0) {
          const double rz = s_tot[0][0], rr = s_tot[1][0];
          if (sc.after_xr(rz, rr, it - 1) && it < iters && !s_abort) {
            sc.advance(rz);
          } else {
            sc.store(sst, it - 1);
            if constexpr (MODE == kPersistMixed) scalar_after_mx_cr(&sst, rz, rr);
            else scalar_after_xr(&sst, rz, rr);
            if (s_abort && sst.status == ST_RUNNING) sst.status = ST_ABORTED;
            s_code[1] = sst.status != ST_RUNNING || MODE == kPersistMixed ? STOP : STOP_AFTER_P;
            sc.beta = sst.beta;
          }
          s_scalar[1] = sc.beta;
        }
      }
#pragma unroll 1
      for (int i = threadIdx.x; i < H; i += blockDim.x) {
        const int h = __ldg(halo + i);
        ld_peer(peer_addr(zs + (h & 0xffff), (unsigned)(h >> 16)), hz[i]);
      }
      __syncthreads();
    } else {
      // z of the halo (published with the partials), then beta
#pragma unroll 1
      for (int ib = threadIdx.x; ib < H; ib += 4 * (int)blockDim.x) {
        ulonglong2 v[4];
        Wait w;
        for (;;) {
          bool ready = true;
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            const int i = ib + m * (int)blockDim.x;
            if (i < H) { v[m] = ld_slot(a.zslot + __ldg(halo + i)); ready = ready && v[m].y == e; }
          }
          if (ready) break;
          if (w.over(a)) { s_failed = 1; break; }
        }
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (ib + m * (int)blockDim.x < H) from_bits(v[m].x, hz[ib + m * (int)blockDim.x]);
      }
      wait_scalar(1, e);
      if (s_failed) break;
    }
    const int code = s_code[1];
    if (code == STOP) break;
    const double beta = s_scalar[1];
#pragma unroll 1
    for (int i = threadIdx.x; i < rows + H; i += blockDim.x) {
      const int j = i < rows ? i : cap + i - rows;
      const V z = i < rows ? zs[i] : hz[i - rows];
      if constexpr (MODE == kPersistMixed) ps[j] = fmaf(float(beta), ps[j], z);
      else if constexpr (MODE == kPersistDf) ps[j] = df::mac(z, df::from_double(beta), ps[j]);
      else ps[j] = fma(beta, ps[j], z);
    }
    __syncthreads();
    if (code != GO) break;
  }

  __syncthreads();
#pragma unroll 1
  for (int i = threadIdx.x; i < rows; i += blockDim.x) {
    wx[row0 + i] = xs[i];
    wr[row0 + i] = rs[i];
    wp[row0 + i] = ps[i];
    if constexpr (MODE == kPersistDouble) s.q[row0 + i] = zs[i];   // z of the iteration that stopped
  }
  if constexpr (CLUSTER) {
    if (cta == 0 && threadIdx.x == 0) {
      sst.coop_epoch += it;
      sst.guard += (it + 3) / 4;
      *s.st = sst;
      tell_done<MODE>(a, sst);
    }
    cluster_barrier();   // no CTA leaves while another may read its shared memory
  }
}

// NC for the sizes of a layout: register rows that cover the CTA's rows, at
// most four; threads per row above 2 (rows of 16 nonzeros and more) keep one.
template <int T, int MODE, bool CL>
const void* kernel_nc(int nc) {
  if constexpr (T <= 2) {
    if (nc >= 3) return (const void*)k_persist<T, MODE, CL, 4>;
    if (nc == 2) return (const void*)k_persist<T, MODE, CL, 2>;
  }
  return (const void*)k_persist<T, MODE, CL, 1>;
}
template <int MODE, bool CL>
const void* kernel_of(int tpr, int nc) {
  switch (tpr) {
    case 1: return kernel_nc<1, MODE, CL>(nc);
    case 2: return kernel_nc<2, MODE, CL>(nc);
    case 4: return kernel_nc<4, MODE, CL>(nc);
    case 8: return kernel_nc<8, MODE, CL>(nc);
    case 16: return kernel_nc<16, MODE, CL>(nc);
    default: return kernel_nc<32, MODE, CL>(nc);
  }
}

}  // namespace
}  // namespace nlgb
