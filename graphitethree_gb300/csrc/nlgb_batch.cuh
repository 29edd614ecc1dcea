// nlgb_batch.cuh -- the persistent kernel that runs many systems in one launch.
// One translation unit for each of its two forms (nlgb_batch.cu, without mixed
// systems, and nlgb_batch_mx.cu): the phase procedures are functions, which a
// translation unit's kernels share together with their allocation of registers.
// In one unit with the FP32 SpMV, which keeps three nonzeros in flight, the
// other phases were slower: a 520 x 500 LSCM system and 12 small ones, 1,500
// iterations, double-float 339 ms (now 282), FP64 358 (351), mixed 262 (243).
//
// Layout of one launch (grid = every co-resident CTA, cooperative launch):
//   * large systems are run by "teams" of k CTAs; a team synchronises its
//     phases with a global-memory barrier (bounded spin, then an error flag),
//     runs the system it was planned for, then draws further large systems
//     from a shared team queue (largest first) until it is empty;
//   * every other CTA is a queue worker: it pops the next small system from
//     an atomic queue and runs it alone (phases separated by __syncthreads).
// Each system's iteration is the same sequence of tile procedures and scalar
// steps as the single-system solver (nlgb_solver.cu), with the same tiles
// and the same canonical reductions, so a system's iterates do not depend on
// the team size, on the other systems in the launch or on where an epoch
// boundary falls: a result is bit-identical alone and in any mix.
// Every CTA of a team computes the scalars redundantly from the tile
// partials; rank 0 stores the system state back to HBM.
#pragma once
#include "nlgb_batch.h"
#include "nlgb_core.cuh"

namespace nlgb {
namespace {

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Barriers this CTA has completed in the current launch (set to 0 at kernel
// start; every CTA of a team passes the same sequence of barriers).
__shared__ unsigned long long s_bar_epoch;
// Limit of one barrier wait (BatchArgs::barrier_timeout_ns, 4 s by default),
// after which the CTA sets the launch's error flag and returns.
__shared__ unsigned long long s_bar_timeout_ns;
// Time box: the CTA's deadline on the GPU clock (0: none) and the stop
// decision of the current iteration of its system.
__shared__ unsigned long long s_deadline;
__shared__ int s_stop;

// Start of an iteration: the team's rank 0 decides whether the time box is
// used up and publishes the answer before the iteration's first barrier (a
// single CTA keeps it in shared memory).
__device__ __forceinline__ void stop_probe(TeamBar* bar, int k, int r) {
  if (s_deadline == 0ULL || r != 0 || threadIdx.x != 0) return;
  const int late = globaltimer_ns() > s_deadline ? 1 : 0;
  if (k > 1) *((volatile unsigned long long*)&bar->stop.count) = (unsigned long long)late;
  else s_stop = late;
}
// Thread 0, after the iteration's first barrier: every CTA of the team reads
// rank 0's decision (the writer passes the barrier's release before any
// reader's acquire; the next write comes after the iteration's last barrier,
// which every reader passes after reading).
__device__ __forceinline__ void stop_read(TeamBar* bar, int k) {
  if (s_deadline != 0ULL && k > 1) s_stop = (int)*((volatile unsigned long long*)&bar->stop.count);
}

__device__ __forceinline__ unsigned long long atom_add_acq_rel(unsigned long long* p, unsigned long long v) {
  unsigned long long old;
  asm volatile("atom.acq_rel.gpu.global.add.u64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory");
  return old;
}

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Team barrier.  k == 1: a CTA barrier.  Returns false (in every thread) if
// the wait timed out or another CTA already flagged an error.  r: rank of
// this CTA in the team.  The __syncthreads before the arrival orders the
// CTA's writes before thread 0's release; thread 0's acquire and the
// __syncthreads after the wait order the other CTAs' writes before this
// CTA's next reads (which go through L2: __ldcg).
__device__ __noinline__ bool team_sync(TeamBar* bar, int k, int r, int* err) {
  if (k == 1) {
    __syncthreads();
    return true;
  }
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    const unsigned long long e = s_bar_epoch + 1;
    s_bar_epoch = e;
    unsigned long long target;
    if (k <= kBarFlat) {
      atom_add_acq_rel(&bar->top.count, 1ULL);
      target = e * (unsigned long long)k;
    } else {
      const int g = r / kBarGroup;
      const int n_groups = (k + kBarGroup - 1) / kBarGroup;
      const unsigned long long g_size = (unsigned long long)min(kBarGroup, k - g * kBarGroup);
      if (atom_add_acq_rel(&bar->grp[g].count, 1ULL) + 1ULL == e * g_size)
        atom_add_acq_rel(&bar->top.count, 1ULL);
      target = e * (unsigned long long)n_groups;
    }
    if (ld_acquire(&bar->top.count) < target) {
      const unsigned long long t0 = globaltimer_ns();
      unsigned int spins = 0;
      while (ld_acquire(&bar->top.count) < target) {
        if ((++spins & 31u) == 0u) {
          if (*((volatile int*)err) != 0) { ok = 0; break; }
          if (globaltimer_ns() - t0 > s_bar_timeout_ns) {
            atomicExch(err, 1);
            ok = 0;
            break;
          }
        }
        __nanosleep(8);
      }
    }
  }
  __syncthreads();
  return ok != 0;
}

// Runtime dispatch of the SpMV tile procedures on the system's threads-per-row
// (coherent gathers: x and p were written earlier in this kernel).
#define NLGB_TPR_SWITCH(...)                                            \
  switch (s.tpr) {                                                      \
    case 1: { constexpr int T = 1; __VA_ARGS__; } break;                \
    case 2: { constexpr int T = 2; __VA_ARGS__; } break;                \
    case 4: { constexpr int T = 4; __VA_ARGS__; } break;                \
    case 8: { constexpr int T = 8; __VA_ARGS__; } break;                \
    case 16: { constexpr int T = 16; __VA_ARGS__; } break;              \
    default: { constexpr int T = 32; __VA_ARGS__; } break;              \
  }

__device__ void put_parts(const SysView& s, int tile, int slot, const double* v, int K) {
  if (threadIdx.x == 0)
    for (int k = 0; k < K; ++k) __stcg(s.part + (size_t)tile * kParts + slot + k, v[k]);
}

template <int K>
__device__ void get_sums(const SysView& s, int slot, double (&o)[K]) {
  int comp[K];
#pragma unroll
  for (int k = 0; k < K; ++k) comp[k] = slot + k;
  canon_reduce<K>(s.part, s.n_tiles, comp, o);
}

// Thread 0 applies a scalar step to the CTA's shared copy of the state; the
// barrier after it publishes the result to the other threads.
#define NLGB_SCALAR(stmt)        \
  if (threadIdx.x == 0) { stmt; } \
  __syncthreads();

// Phase procedures: the tile loop of one phase for this CTA's tiles (t = r,
// r + k, ...), partials stored for the canonical reduction.  Kept out of line
// so that each is register-allocated on its own: inlined into the one
// persistent kernel (six threads-per-row variants of each) they forced the
// kernel to spill inside the SpMV loops.  NLGB_HOT_PHASE marks the three
// phases of the FP64 iteration.
#ifndef NLGB_HOT_PHASE
#define NLGB_HOT_PHASE __noinline__
#endif
template <bool D>
__device__ __noinline__ void ph_residual(const SysView& s, int r, int k) {
  for (int t = r; t < s.n_tiles; t += k) {
    double v[3];
    NLGB_TPR_SWITCH((phase_residual<D, T, true>(s, t, v)));
    put_parts(s, t, kSlotInit, v, 3);
  }
}
__device__ __noinline__ void ph_mx_outer(const SysView& s, int r, int k) {
  for (int t = r; t < s.n_tiles; t += k) {
    double v[4];
    NLGB_TPR_SWITCH(tile_mx_outer<T, true>(s, t, v));
    put_parts(s, t, kSlotInit, v, 4);
  }
}
template <bool D>
__device__ NLGB_HOT_PHASE void ph_spmv_pq(const SysView& s, int r, int k) {
  for (int t = r; t < s.n_tiles; t += k) {
    double v[1];
    NLGB_TPR_SWITCH((v[0] = phase_spmv_pq<D, T, true>(s, t)));
    put_parts(s, t, kSlotPQ, v, 1);
  }
}
template <bool D>
__device__ NLGB_HOT_PHASE void ph_update_xr(const SysView& s, int r, int k, double alpha) {
  for (int t = r; t < s.n_tiles; t += k) {
    double v[2];
    phase_update_xr<D>(s, t, alpha, v);
    put_parts(s, t, kSlotXR, v, 2);
  }
}
template <bool D>
__device__ NLGB_HOT_PHASE void ph_update_p(const SysView& s, int r, int k, double beta) {
  for (int t = r; t < s.n_tiles; t += k) phase_update_p<D>(s, t, beta);
}
__device__ __noinline__ void ph_mx_update_p(const SysView& s, int r, int k, double beta) {
  for (int t = r; t < s.n_tiles; t += k) tile_mx_update_p(s, t, beta);
}
__device__ __noinline__ void ph_mx_spmv_pq(const SysView& s, int r, int k) {
  for (int t = r; t < s.n_tiles; t += k) {
    double v[1];
    NLGB_TPR_SWITCH(v[0] = tile_mx_spmv_pq<T, true>(s, t));
    put_parts(s, t, kSlotPQ, v, 1);
  }
}
__device__ __noinline__ void ph_mx_update_cr(const SysView& s, int r, int k, double alpha) {
  for (int t = r; t < s.n_tiles; t += k) {
    double v[2];
    tile_mx_update_cr(s, t, alpha, v);
    put_parts(s, t, kSlotXR, v, 2);
  }
}
__device__ __noinline__ void ph_mx_apply(const SysView& s, int r, int k) {
  for (int t = r; t < s.n_tiles; t += k) tile_mx_apply(s, t);
}
template <bool D>
__device__ __noinline__ void ph_final(const SysView& s, int r, int k, bool zero_rhs) {
  for (int t = r; t < s.n_tiles; t += k) {
    double v[1] = {0.0};
    if (zero_rhs) {
      tile_zero_x(s, t);
    } else {
      NLGB_TPR_SWITCH((v[0] = phase_true_rr<D, T, true>(s, t)));
    }
    put_parts(s, t, kSlotFinal, v, 1);
  }
}

// Canonical sums of K consecutive partial slots (out of line, as above).
struct Sums4 { double v[4]; };
__device__ __noinline__ Sums4 sums_of(const SysView& s, int slot, int K) {
  Sums4 o = {{0.0, 0.0, 0.0, 0.0}};
  switch (K) {
    case 1: { double a[1]; get_sums<1>(s, slot, a); o.v[0] = a[0]; } break;
    case 2: { double a[2]; get_sums<2>(s, slot, a); o.v[0] = a[0]; o.v[1] = a[1]; } break;
    case 3: { double a[3]; get_sums<3>(s, slot, a); for (int i = 0; i < 3; ++i) o.v[i] = a[i]; } break;
    default: { double a[4]; get_sums<4>(s, slot, a); for (int i = 0; i < 4; ++i) o.v[i] = a[i]; } break;
  }
  return o;
}

// One system, run by a team (rank r of k CTAs) for at most `budget`
// iterations.  st: the CTA's shared-memory copy of the system state.  MX: it may
// be a mixed one.
template <bool MX>
__device__ void run_system_once(const SysView& s, SysState* st, int r, int k, TeamBar* bar, int* err,
                                long long budget) {
  const bool mixed = MX && st->precision == 1;
  long long done_iters = 0;
  if (st->stage == 0) {
    if (!mixed) {
      if (s.df) ph_residual<true>(s, r, k);
      else ph_residual<false>(s, r, k);
      if (!team_sync(bar, k, r, err)) { NLGB_SCALAR(st->status = ST_DEVICE_ERR; st->stage = 3); return; }
      const Sums4 o = sums_of(s, kSlotInit, 3);
      NLGB_SCALAR(scalar_after_init(st, o.v[0], o.v[1], o.v[2]); st->stage = st->status == ST_RUNNING ? 1 : 2);
    } else {
      // initial FP64 residual (first "reliable update"; c = 0, p = 0)
      ph_mx_outer(s, r, k);
      if (!team_sync(bar, k, r, err)) { NLGB_SCALAR(st->status = ST_DEVICE_ERR; st->stage = 3); return; }
      const Sums4 o = sums_of(s, kSlotInit, 4);
      NLGB_SCALAR(st->mode = 0; scalar_after_outer(st, o.v[0], o.v[1], o.v[2], o.v[3]);
                  st->stage = st->status == ST_RUNNING ? 1 : 2);
    }
  }
  for (;;) {
    if (st->stage == 4) {
      // continuation after a failed true-residual check (possibly left by
      // another executor): the pending p update, then more iterations
      if (s.df) ph_update_p<true>(s, r, k, st->beta);
      else ph_update_p<false>(s, r, k, st->beta);
      if (!team_sync(bar, k, r, err)) { NLGB_SCALAR(st->status = ST_DEVICE_ERR; st->stage = 3); return; }
      NLGB_SCALAR(st->stage = 1);
    }
    while (st->stage == 1 && (budget <= 0 || done_iters < budget)) {
      stop_probe(bar, k, r);
      if (!mixed) {
        // q = A p, p.q
        if (s.df) ph_spmv_pq<true>(s, r, k);
        else ph_spmv_pq<false>(s, r, k);
        if (!team_sync(bar, k, r, err)) break;
        {
          const Sums4 o = sums_of(s, kSlotPQ, 1);
          NLGB_SCALAR(scalar_after_pq(st, o.v[0]); stop_read(bar, k));
        }
        if (st->status != ST_RUNNING) { NLGB_SCALAR(st->stage = 2); break; }
        if (s.df) ph_update_xr<true>(s, r, k, st->alpha);
        else ph_update_xr<false>(s, r, k, st->alpha);
        if (!team_sync(bar, k, r, err)) break;
        {
          const Sums4 o = sums_of(s, kSlotXR, 2);
          NLGB_SCALAR(scalar_after_xr(st, o.v[0], o.v[1]));
        }
        ++done_iters;
        if (st->status != ST_RUNNING) { NLGB_SCALAR(st->stage = 2); break; }
        if (s.df) ph_update_p<true>(s, r, k, st->beta);
        else ph_update_p<false>(s, r, k, st->beta);
        if (!team_sync(bar, k, r, err)) break;
        if (s_stop) break;   // time box used up: the system resumes next epoch
      } else {
        // FP32 PCG iteration with FP64 reliable updates; same phase order as
        // the graph solver: p update, SpMV + p.q, c/r update, [update].
        ph_mx_update_p(s, r, k, st->beta);
        if (!team_sync(bar, k, r, err)) break;
        ph_mx_spmv_pq(s, r, k);
        if (!team_sync(bar, k, r, err)) break;
        {
          const Sums4 o = sums_of(s, kSlotPQ, 1);
          NLGB_SCALAR(scalar_after_pq(st, o.v[0]); stop_read(bar, k));
        }
        if (st->status != ST_RUNNING) { NLGB_SCALAR(st->stage = 2); break; }
        ph_mx_update_cr(s, r, k, st->alpha);
        if (!team_sync(bar, k, r, err)) break;
        {
          const Sums4 o = sums_of(s, kSlotXR, 2);
          NLGB_SCALAR(scalar_after_mx_cr(st, o.v[0], o.v[1]));
        }
        ++done_iters;
        if (st->status != ST_RUNNING) { NLGB_SCALAR(st->stage = 2); break; }
        if (st->mode == 0) {
          // reliable update: x += c, r = b - A x in FP64, FP32 residual replaced
          ph_mx_apply(s, r, k);
          if (!team_sync(bar, k, r, err)) break;
          ph_mx_outer(s, r, k);
          if (!team_sync(bar, k, r, err)) break;
          const Sums4 o = sums_of(s, kSlotInit, 4);
          NLGB_SCALAR(scalar_after_outer(st, o.v[0], o.v[1], o.v[2], o.v[3]);
                      // FP32 cannot track this system: continue it in FP64
                      // from the current x (same rule as the graph solver).
                      if (st->status == ST_STAGNATION && !st->fell_back) {
                        st->status = ST_RUNNING; st->precision = 0; st->fell_back = 1;
                        st->stage = 0; st->mode = 0; st->iter_at_fallback = st->iter;
                      });
          if (st->stage == 0) break;
          if (st->status != ST_RUNNING) { NLGB_SCALAR(st->stage = 2); break; }
        }
        if (s_stop) break;   // time box used up: the system resumes next epoch
      }
    }
    if (*((volatile int*)err) != 0 && st->stage != 3) {
      NLGB_SCALAR(st->status = ST_DEVICE_ERR; st->stage = 3);
      return;
    }
    if (st->stage == 2) {
      // final true residual (FP64) of the returned x; x = 0 when b == 0
      if (s.df) ph_final<true>(s, r, k, st->zero_rhs != 0);
      else ph_final<false>(s, r, k, st->zero_rhs != 0);
      if (!team_sync(bar, k, r, err)) { NLGB_SCALAR(st->status = ST_DEVICE_ERR; st->stage = 3); return; }
      const Sums4 o = sums_of(s, kSlotFinal, 1);
      NLGB_SCALAR(st->rr_true = o.v[0]; st->stage = scalar_after_check(st) ? 4 : 3);
      if (st->stage == 4) continue;
    }
    return;
  }
}

// One system; a mixed system that falls back to FP64 restarts here at stage
// 0 with precision 0 (its FP32 iterations stay counted).
template <bool MX>
__device__ void run_system(const SysView& s, SysState* st, int r, int k, TeamBar* bar, int* err,
                           long long budget) {
  run_system_once<MX>(s, st, r, k, bar, err, budget);
  if (MX && st->stage == 0 && st->fell_back && st->precision == 0)
    run_system_once<MX>(s, st, r, k, bar, err, budget);
}

// Four CTAs per SM (64 registers): stating the bound lets ptxas plan for it,
// with far fewer spills than its own choice of the same 64 registers.  MX: with
// mixed systems.
template <bool MX>
__global__ void __launch_bounds__(kCTA, 4) k_batch(BatchArgs a) {
  __shared__ SysView sv;
  __shared__ SysState sst;
  __shared__ int pick;
  const int cta = blockIdx.x;
  if (threadIdx.x == 0) {
    s_bar_epoch = 0ULL;
    s_bar_timeout_ns = a.barrier_timeout_ns;
    s_deadline = a.epoch_ns > 0ULL ? globaltimer_ns() + a.epoch_ns : 0ULL;
    s_stop = 0;
  }
  if (a.times && cta == 0 && threadIdx.x == 0) a.times[0] = globaltimer_ns();
  __syncthreads();
  auto load = [&](int sys) {
    if (threadIdx.x == 0) {
      sv = a.views[sys];
      sst = *sv.st;
      s_stop = 0;
    }
    __syncthreads();
  };
  auto past_deadline = [&]() { return s_deadline != 0ULL && globaltimer_ns() > s_deadline; };
  auto store = [&](bool rank0) {
    __syncthreads();
    if (rank0 && threadIdx.x == 0) {
      *sv.st = sst;
      __threadfence();
    }
    __syncthreads();
  };
  if (cta < a.team_ctas) {
    const int team = a.cta_team[cta];
    const TeamDesc td = a.teams[team];
    const int r = cta - td.cta_begin;
    TeamBar* bar = a.bars + team;
    for (int j = td.sys_begin; j < td.sys_end; ++j) {
      load(a.team_sys[j]);
      if (sst.stage != 3) run_system<MX>(sv, &sst, r, td.k, bar, a.err, sv.budget > 0 ? sv.budget : a.budget);
      store(r == 0);
    }
    // Then the shared team queue: rank 0 draws the next system and publishes
    // it through the team barrier; a second barrier keeps the next draw from
    // overwriting `pick` before every CTA of the team has read it.
    while (a.n_tqueue > 0) {
      // past the time box, rank 0 draws nothing (publishes the end of the queue)
      if (r == 0 && threadIdx.x == 0)
        *((volatile unsigned long long*)&bar->pick.count) =
            past_deadline() ? (unsigned long long)a.n_tqueue : atomicAdd(a.tqueue_head, 1u);
      if (!team_sync(bar, td.k, r, a.err)) break;
      if (threadIdx.x == 0) pick = (int)*((volatile unsigned long long*)&bar->pick.count);
      __syncthreads();
      const int q = pick;
      if (!team_sync(bar, td.k, r, a.err)) break;
      if (q >= a.n_tqueue) break;
      load(a.tqueue[q]);
      if (sst.stage != 3) run_system<MX>(sv, &sst, r, td.k, bar, a.err, sv.budget > 0 ? sv.budget : a.budget);
      store(r == 0);
    }
    if (a.times && r == 0 && threadIdx.x == 0) a.times[2 + team] = globaltimer_ns();
  } else {
    while (true) {
      if (threadIdx.x == 0) pick = past_deadline() ? a.n_queue : (int)atomicAdd(a.queue_head, 1u);
      __syncthreads();
      const int q = pick;
      __syncthreads();
      if (q >= a.n_queue) break;
      load(a.queue[q]);
      if (sst.stage != 3) run_system<MX>(sv, &sst, 0, 1, nullptr, a.err, sv.budget > 0 ? sv.budget : a.budget);
      store(true);
    }
    if (a.times && threadIdx.x == 0) atomicMax(&a.times[1], globaltimer_ns());
  }
}

}  // namespace
}  // namespace nlgb
