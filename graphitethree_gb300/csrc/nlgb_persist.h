// nlgb_persist.h -- the persistent single-system PCG kernel (nlgb_persist.cu).
#pragma once
#include <cuda_runtime.h>

#include "nlgb_core.cuh"
#include "nlgb_internal.h"

namespace nlgb {

enum { kPersistDouble = 0, kPersistDf = 1, kPersistMixed = 2 };

constexpr int kPersistBlock = 512;        // threads per CTA at most (128 registers each)
constexpr int kPersistSlots = 9;          // tiles per CTA at most (1,216 tiles on 151 CTAs)
// The cluster form: up to 16 CTAs, whose exchanges cost less than the grid form's.
// Tiles that share a CTA cost more the more nonzeros they have, above all with long
// rows, which a CTA reads from L2.  So rows of more than two threads take the grid
// from 17 tiles on (where the system has the GPU to itself, or they are long), rows
// of two (LSCM) from 33 on where it has, others from 65 on.  Sharing the GPU: 4
// charts of 60 to 128 vertices a side at once 15.0 ms, with grids from 17 on 16.9.
// us per iteration, cluster -> grid (FP64; mixed):
//   fairing  17 tiles 5.2 -> 6.2; 5.5 -> 6.8    32  5.6 -> 5.7; 5.8 -> 5.9
//            48       6.3 -> 6.0; 6.0 -> 6.3    64  6.8 -> 6.3; 6.3 -> 6.3
//   LSCM     17       5.9 -> 6.5; 4.7 -> 5.9    32  6.3 -> 6.1; 5.0 -> 5.7
//            33       6.8 -> 6.2; 5.2 -> 5.4    64  8.1 -> 6.2; 5.8 -> 5.6
//   64 tiles of rows of 24 nonzeros 22.6 -> 11.2, of 92 42.2 -> 16.5, of 356 105.9 ->
//   35.7 (one cooperative kernel per iteration 22.4, 32.5, 69.5)
constexpr int kPersistCluster = 16;
constexpr int kPersistClusterTiles = 64;  // with four tiles on each
// Nonzeros of a CTA's tiles where rows have more than two threads (of which one
// row per lane group stays in registers): above, fewer tiles per CTA.  6,000 rows
// of 46 nonzeros, 17,400 per CTA: 22.5 us per iteration (25.0 in the cooperative
// kernel); 8,000 of 47, 23,500: 27.5 (24.9).
constexpr long long kPersistCtaNnz = 16384;
constexpr int kPersistRed = 8 * 36;       // 8-byte words of one staged value of a tile

// How a launch left its system: running, at a reliable update, or stopped.
enum PersistEnd : unsigned { kPersistPaused = 0, kPersistUpdate = 1, kPersistStopped = 2 };

struct PersistArgs {
  SysView s;
  ulonglong2* slot;            // grid form: 3 x n_tiles, p.q, r.z, r.r of every tile as (value, epoch)
  ulonglong2* ctl;             // grid form: [0] alpha, [8] beta as (value, 256 epoch + code)
  ulonglong2* zslot;           // grid form: z of every row as (value, epoch)
  int* err;                    // nonzero: a wait ran out
  unsigned long long wait_ns;  // limit of one wait (persist_launch)
  PersistLayout lay;
  long long iters;             // iterations of this launch at most (fewer where the chunk's budget ends)
  unsigned int* done;          // host-mapped, or null: done_value + a PersistEnd when the launch ends
  unsigned int done_value;
};

// Exchange area (zeroed before a solve): partial slots, control slots, z
// slots, the error word.
inline size_t persist_bytes(int n, int n_tiles) {
  return ((size_t)3 * n_tiles + 16 + (size_t)n + 1) * sizeof(ulonglong2);
}
inline void persist_bind(PersistArgs& a, void* exch) {
  a.slot = reinterpret_cast<ulonglong2*>(exch);
  a.ctl = a.slot + (size_t)3 * a.s.n_tiles;
  a.zslot = a.ctl + 16;
  a.err = reinterpret_cast<int*>(a.zslot + a.s.n);
}
// Tiles per CTA of a system that shares the GPU: a CTA takes about 5 us per
// iteration and 1.2 us more for every tile, so more tiles use fewer SMs per
// system and fewer tiles finish one sooner.  24 requests of 1k to 20k vertices
// with 2, 3, 4 and 6 tiles: 106, 80, 71, 66 ms; 6 requests of 1k to 4k: 8.4,
// 8.5, 8.8, 10.4 ms.
constexpr int kSharedTiles = 4, kPersistAlone = 0;
// SMs that one system leaves free on a server: for a cluster beside it, and for
// the kernels of admissions (an admission waits for a dozen of them one after
// the other, and a CTA of k_persist has its SM's registers to itself).  Several
// systems together may take all SMs: their chunks end at different times, and
// with seven SMs always free two systems of 20k vertices no longer ran side by
// side (24 requests of 1k to 20k vertices 65 -> 73 ms).  Latency of a request of 1.6k vertices beside an
// LSCM system of 157k unknowns, with all SMs taken -> so: 19.4 -> 2.2 ms.
constexpr int kSharedLeave = kPersistCluster + 7;
// CTAs that own a system's tiles, with per_cta tiles on each (kPersistAlone: one,
// the system has the GPU to itself), fewer where rows are long, or as many as
// there have to be.  leave > 0: on all but so many SMs (where nine tiles per CTA
// allow that), and the fewest CTAs with as many tiles on the busiest.
int persist_ctas(const DeviceCRS& A, int n_tiles, int per_cta, int sms, int leave = 0);
// The same without a look at the rows; spread: a grid rather than more tiles than
// per_cta on the CTAs of a cluster.
int persist_ctas_for(int n_tiles, int per_cta, int sms, int leave = 0, bool spread = false);
// About the time of an iteration of a system that shares the GPU, us.
double persist_iteration_us(int n_tiles, int ctas);
// Launches the kernel.  Environment: NLGB_BARRIER_TIMEOUT_MS limits its waits
// (4 s).  For tests: NLGB_TEST_PERSIST_SHORTFALL=1 leaves out the CTA of the grid
// form that publishes alpha and beta, so that waits run out;
// NLGB_TEST_PERSIST_REFUSE=n refuses the launches from the n-th one on.
cudaError_t persist_launch(const PersistPlan& p, const PersistArgs& a, cudaStream_t s);
// The kernel for a layout (nlgb_persist_*.cu): nc rows per lane group in registers.
const void* persist_kernel_f64(int tpr, bool cluster, int nc);
const void* persist_kernel_df(int tpr, bool cluster, int nc);
const void* persist_kernel_mx(int tpr, bool cluster, int nc);

}  // namespace nlgb
