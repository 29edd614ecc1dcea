// nlgb_batch.cu -- many independent Jacobi-PCG systems in one persistent
// kernel launch (plain FP64 or mixed FP32/FP64 per system), or, where all of
// them fit it and they are few enough, each on the persistent single-system
// kernel (persist_batch).
//
// Reference context: geogram's mesh_make_atlas solves one LSCM system per
// chart, one after another, each through nlSolve (called from
// src/lib/OGF/mesh/commands/mesh_grob_surface_commands.cpp:724); a GPU that
// runs them one at a time is launch- and latency-bound on the small charts.
//
// The batched kernel itself is in nlgb_batch.cuh.
#include "nlgb_batch.cuh"
#include "nlgb_batch.h"
#include "nlgb_core.cuh"
#include "nlgb_internal.h"
#include "nlgb_persist.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <numeric>

namespace nlgb {

static size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

// Small pinned allocations share a chunk of the driver's: to map the first one
// and to give the last one back takes 0.3 ms.  64 bytes stay, so that a batch does
// not pay that (a call with one small system 0.55 -> 0.24 ms).
void keep_pinned_chunk() {
  static const bool kept = [] {
    void* p = nullptr;
    const bool ok = cudaMallocHost(&p, 64) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok;
  }();
  (void)kept;
}

namespace {

// A batch on the persistent single-system kernel: systems at a time, iterations
// of one launch, and the rule it is chosen by (persist_batch_pays).
constexpr int kPersistLanes = 32;
constexpr long long kPersistBatchIters = 1024;
constexpr double kPersistBatchRatio = 0.5;

__global__ void k_gather_states(const SysView* views, int n, SysState* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = *views[i].st;
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
BatchRunner::~BatchRunner() {
  cudaFree(d_views_); cudaFree(d_teams_); cudaFree(d_cta_team_); cudaFree(d_team_sys_);
  cudaFree(d_queue_); cudaFree(d_tqueue_); cudaFree(d_bars_); cudaFree(d_ctl_); cudaFree(d_times_);
  if (h_err_) cudaFreeHost(h_err_);
  cudaFree(d_states_);
  if (ev0_) cudaEventDestroy(ev0_);
  if (ev1_) cudaEventDestroy(ev1_);
}

cudaError_t BatchRunner::init(cudaStream_t s) {
  stream_ = s;
  int dev = 0;
  NLGB_CUDA_TRY(cudaGetDevice(&dev));
  NLGB_CUDA_TRY(cudaDeviceGetAttribute(&n_sm_, cudaDevAttrMultiProcessorCount, dev));
  int per_sm = 0, per_sm_mx = 0;
  NLGB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<false>, kCTA, 0));
  NLGB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_mx, batch_kernel_mixed(), kCTA, 0));
  per_sm_ = std::max(1, std::min(per_sm, per_sm_mx));
  grid_ = n_sm_ * per_sm_;
  NLGB_CUDA_TRY(cudaMalloc(&d_ctl_, 3 * sizeof(int)));
  keep_pinned_chunk();
  NLGB_CUDA_TRY(cudaMallocHost(&h_err_, sizeof(int)));
  *h_err_ = 0;
  NLGB_CUDA_TRY(cudaEventCreate(&ev0_));
  NLGB_CUDA_TRY(cudaEventCreate(&ev1_));
  // Test hooks for the barrier's failure path (read once per runner): a
  // shorter wait limit, and a first team told to wait for one CTA more than
  // it is given, so that its first barrier runs out -- the kernel must then
  // flag the error, return, and leave the GPU usable.
  if (const char* e = std::getenv("NLGB_BARRIER_TIMEOUT_MS")) {
    const double ms = std::atof(e);
    if (ms > 0.0) barrier_timeout_ns_ = (unsigned long long)(ms * 1e6);
  }
  if (const char* e = std::getenv("NLGB_TEST_TEAM_SHORTFALL")) test_shortfall_ = e[0] == '1';
  return cudaSuccess;
}

template <typename T>
static cudaError_t ensure(T*& p, size_t& cap, size_t n) {
  if (n <= cap && p) return cudaSuccess;
  cudaFree(p);
  p = nullptr;
  cap = std::max<size_t>(n, 16);
  return cudaMalloc(&p, cap * sizeof(T));
}

// Schedule for one launch.  Small systems (fewer than kLargeTiles tiles) go to
// the single-CTA queue, whose workers get a share of the grid proportional to
// the small systems' work (at least one, at most one per system).  The large
// ones, largest first, get teams sized by their share of the remaining CTAs
// (at least 2, at most one CTA per tile) until the CTAs run out; the rest
// wait in the team queue, from which every team draws (largest first) once
// its own system is done -- list scheduling, so one mis-estimated system
// does not leave the other teams idle.
void BatchRunner::plan(const std::vector<SysView>& views, const std::vector<long long>& work) {
  teams_.clear(); cta_team_.clear(); team_sys_.clear(); queue_.clear(); tqueue_.clear();
  const int n = (int)views.size();
  std::vector<int> order(n);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return work[a] > work[b]; });
  std::vector<int> large;
  double w_large = 0.0, w_small = 0.0;
  for (int i : order) {
    const double w = (double)std::max(1LL, work[i]);
    if (views[i].n_tiles >= kLargeTiles) { large.push_back(i); w_large += w; }
    else { queue_.push_back(i); w_small += w; }
  }
  if (large.empty()) return;
  int reserve = 0;
  if (!queue_.empty()) {
    reserve = (int)std::ceil((double)grid_ * w_small / (w_small + w_large));
    reserve = std::max(1, std::min(reserve, std::min((int)queue_.size(), grid_ / 2)));
  }
  const int avail = grid_ - reserve_ - reserve;
  if (avail < 2) {   // no room for a team: everything goes to the queue workers
    queue_.insert(queue_.begin(), large.begin(), large.end());
    return;
  }
  const double per_cta = w_large / (double)avail;
  int cta = 0;
  for (int i : large) {
    const double w = (double)std::max(1LL, work[i]);
    const int cap = std::min(kBarGroup * kBarMaxGroups, std::max(2, views[i].n_tiles));
    int k = (int)std::min<double>((double)cap, std::max(2.0, std::floor(w / per_cta)));
    if (cta + k > avail) k = avail - cta;     // the last team takes what is left
    if (k < 2) { tqueue_.push_back(i); continue; }
    // Balanced: the fewest CTAs with the same tiles on the busiest CTA (1,023
    // tiles on 604 CTAs are 2 on the busiest, as on 512; the other 92 CTAs
    // would only add barrier and reduction traffic).
    const int per = (views[i].n_tiles + k - 1) / k;
    k = std::max(2, (views[i].n_tiles + per - 1) / per);
    TeamDesc td;
    td.cta_begin = cta;
    td.k = k;
    td.sys_begin = (int)team_sys_.size();
    team_sys_.push_back(i);
    td.sys_end = (int)team_sys_.size();
    for (int c = 0; c < k; ++c) cta_team_.push_back((int)teams_.size());
    teams_.push_back(td);
    cta += k;
  }
}

constexpr int kPrioTilesPerCta = 4;

void BatchRunner::plan_priority(const std::vector<SysView>& views) {
  teams_.clear(); cta_team_.clear(); team_sys_.clear(); queue_.clear(); tqueue_.clear();
  const int n = (int)views.size();
  const int avail_all = std::max(1, grid_ - reserve_);
  int n_small = 0;
  for (int i = 0; i < n; ++i) n_small += views[i].n_tiles < kLargeTiles ? 1 : 0;
  // queue workers: one per small system, at most half the grid
  const int workers = n_small == 0 ? 0 : std::max(1, std::min(n_small, avail_all / 2));
  const int avail = avail_all - workers;
  int cta = 0;
  for (int i = 0; i < n; ++i) {
    if (views[i].n_tiles < kLargeTiles) { queue_.push_back(i); continue; }
    const int room = avail - cta;
    if (room < 2) { tqueue_.push_back(i); continue; }
    // about kPrioTilesPerCta tiles per CTA: enough CTAs to finish the
    // system soon, few enough that each CTA's tile work outweighs the
    // team's barriers and that the next systems get teams too
    int k = std::min({(views[i].n_tiles + kPrioTilesPerCta - 1) / kPrioTilesPerCta, kBarGroup * kBarMaxGroups,
                      room});
    k = std::max(2, k);
    // balanced: the fewest CTAs with the same tiles on the busiest CTA
    const int per = (views[i].n_tiles + k - 1) / k;
    k = std::max(2, (views[i].n_tiles + per - 1) / per);
    TeamDesc td;
    td.cta_begin = cta;
    td.k = k;
    td.sys_begin = (int)team_sys_.size();
    team_sys_.push_back(i);
    td.sys_end = (int)team_sys_.size();
    for (int c = 0; c < k; ++c) cta_team_.push_back((int)teams_.size());
    teams_.push_back(td);
    cta += k;
  }
  // without any team, large systems left over go to the queue workers too
  if (teams_.empty() && !tqueue_.empty()) {
    queue_.insert(queue_.end(), tqueue_.begin(), tqueue_.end());
    tqueue_.clear();
  }
}

cudaError_t BatchRunner::run(const std::vector<SysView>& views, const std::vector<long long>& work,
                             long long budget, BatchLaunchStats* stats) {
  NLGB_CUDA_TRY(launch(views, work, budget));
  return finish(stats);
}

cudaError_t BatchRunner::launch(const std::vector<SysView>& views, const std::vector<long long>& work,
                                long long budget) {
  pending_ = false;
  if (views.empty()) return cudaSuccess;
  if (priority_plan_) plan_priority(views);
  else plan(views, work);
  NLGB_CUDA_TRY(ensure(d_views_, cap_views_, views.size()));
  NLGB_CUDA_TRY(ensure(d_teams_, cap_teams_, teams_.size()));
  NLGB_CUDA_TRY(ensure(d_cta_team_, cap_cta_team_, cta_team_.size()));
  NLGB_CUDA_TRY(ensure(d_team_sys_, cap_team_sys_, team_sys_.size()));
  NLGB_CUDA_TRY(ensure(d_queue_, cap_queue_, queue_.size()));
  NLGB_CUDA_TRY(ensure(d_tqueue_, cap_tqueue_, tqueue_.size()));
  NLGB_CUDA_TRY(ensure(d_bars_, cap_bars_, teams_.size()));
  cudaStream_t s = stream_;
  NLGB_CUDA_TRY(cudaMemcpyAsync(d_views_, views.data(), views.size() * sizeof(SysView), cudaMemcpyHostToDevice, s));
  if (!teams_.empty()) {
    if (test_shortfall_ && teams_[0].k < kBarFlat) {
      std::vector<TeamDesc> t = teams_;
      t[0].k += 1;   // no CTA is mapped to the extra rank: the team's barrier cannot complete
      NLGB_CUDA_TRY(cudaMemcpy(d_teams_, t.data(), t.size() * sizeof(TeamDesc), cudaMemcpyHostToDevice));
    } else {
      NLGB_CUDA_TRY(cudaMemcpyAsync(d_teams_, teams_.data(), teams_.size() * sizeof(TeamDesc),
                                    cudaMemcpyHostToDevice, s));
    }
    NLGB_CUDA_TRY(cudaMemcpyAsync(d_cta_team_, cta_team_.data(), cta_team_.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    NLGB_CUDA_TRY(cudaMemcpyAsync(d_team_sys_, team_sys_.data(), team_sys_.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    NLGB_CUDA_TRY(cudaMemsetAsync(d_bars_, 0, teams_.size() * sizeof(TeamBar), s));
  }
  if (!queue_.empty())
    NLGB_CUDA_TRY(cudaMemcpyAsync(d_queue_, queue_.data(), queue_.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  if (!tqueue_.empty())
    NLGB_CUDA_TRY(cudaMemcpyAsync(d_tqueue_, tqueue_.data(), tqueue_.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  NLGB_CUDA_TRY(cudaMemsetAsync(d_ctl_, 0, 3 * sizeof(int), s));
  BatchArgs a;
  std::memset(&a, 0, sizeof(a));
  a.views = d_views_;
  a.teams = d_teams_;
  a.cta_team = d_cta_team_;
  a.team_sys = d_team_sys_;
  a.queue = d_queue_;
  a.tqueue = d_tqueue_;
  a.bars = d_bars_;
  a.err = d_ctl_;
  a.queue_head = reinterpret_cast<unsigned int*>(d_ctl_ + 1);
  a.tqueue_head = reinterpret_cast<unsigned int*>(d_ctl_ + 2);
  a.team_ctas = (int)cta_team_.size();
  a.n_queue = (int)queue_.size();
  a.n_tqueue = teams_.empty() ? 0 : (int)tqueue_.size();
  a.budget = budget;
  a.times = nullptr;
  a.barrier_timeout_ns = barrier_timeout_ns_;
  a.epoch_ns = epoch_ns_;
  if (timing_) {
    NLGB_CUDA_TRY(ensure(d_times_, cap_times_, teams_.size() + 2));
    NLGB_CUDA_TRY(cudaMemsetAsync(d_times_, 0, (teams_.size() + 2) * sizeof(unsigned long long), s));
    a.times = d_times_;
  }
  // Grid: every team CTA plus queue workers, never more than can be resident
  // (less the reserve).
  const int workers = queue_.empty() ? 0 : std::max(1, std::min(std::max(1, grid_ - reserve_) - a.team_ctas,
                                                                (int)queue_.size()));
  const int grid = a.team_ctas + std::max(0, workers);
  void* args[] = {&a};
  NLGB_CUDA_TRY(cudaEventRecord(ev0_, s));
  const bool mixed = std::any_of(views.begin(), views.end(), [](const SysView& v) { return v.r32 != nullptr; });
  const void* kernel = mixed ? batch_kernel_mixed() : (const void*)k_batch<false>;
  NLGB_CUDA_TRY(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kCTA), args, 0, s));
  NLGB_CUDA_TRY(cudaEventRecord(ev1_, s));
  NLGB_CUDA_TRY(cudaMemcpyAsync(h_err_, d_ctl_, sizeof(int), cudaMemcpyDeviceToHost, s));
  last_grid_ = grid;
  last_workers_ = workers;
  pending_ = true;
  return cudaSuccess;
}

cudaError_t BatchRunner::finish(BatchLaunchStats* stats) {
  if (!pending_) {
    if (stats) *stats = BatchLaunchStats();
    return cudaSuccess;
  }
  pending_ = false;
  NLGB_CUDA_TRY(cudaStreamSynchronize(stream_));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ev0_, ev1_);
  if (timing_) {
    h_times_.assign(teams_.size() + 2, 0ULL);
    NLGB_CUDA_TRY(cudaMemcpy(h_times_.data(), d_times_, h_times_.size() * sizeof(unsigned long long),
                             cudaMemcpyDeviceToHost));
  }
  const int err = *h_err_;
  if (stats) {
    stats->ms = ms;
    stats->n_teams = (int)teams_.size();
    stats->team_ctas = (int)cta_team_.size();
    stats->queue_ctas = last_workers_;
    stats->error = err;
    stats->grid = last_grid_;
  }
  if (err) {
    set_error("batched solve: a team barrier timed out");
    return cudaErrorLaunchTimeout;
  }
  return cudaSuccess;
}

cudaError_t BatchRunner::gather_states(SysState* out, int n) {
  if (n <= 0) return cudaSuccess;
  NLGB_CUDA_TRY(ensure(d_states_, cap_states_, (size_t)n));
  k_gather_states<<<(n + 127) / 128, 128, 0, stream_>>>(d_views_, n, d_states_);
  count_launches(1);
  NLGB_CUDA_TRY(cudaGetLastError());
  NLGB_CUDA_TRY(cudaMemcpyAsync(out, d_states_, sizeof(SysState) * n, cudaMemcpyDeviceToHost, stream_));
  NLGB_CUDA_TRY(cudaStreamSynchronize(stream_));
  return cudaSuccess;
}

// ---------------------------------------------------------------------------
// A batch on the persistent single-system kernel.
// ---------------------------------------------------------------------------
namespace {

int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    cudaGetLastError();
  return sms;
}

// Expected time of a system there, up to a factor: iterations of a Jacobi-CG on
// a surface (sqrt(n)) times the time of one.
double persist_time(const SysView& v, int n_sm) {
  return std::sqrt((double)v.n) * persist_iteration_us(v.n_tiles, persist_ctas_for(v.n_tiles, kSharedTiles, n_sm));
}

}  // namespace

// The host starts one system there in about 35 us and builds a matrix's tables
// in 15, while the batched kernel runs up to four systems per SM from one
// launch.  So the line lies at the number of systems in the time of the
// longest one.  LSCM charts, log-uniform long sides, whole call, ms, batched
// kernel -> here with the tables built (first call), and that ratio:
//   40 of 16..128      56.7 -> 27.6 (39.1)    0.03
//   100 of 16..128    105.3 -> 59.7 (62.7)    0.07
//   300 of 16..128    267.5 -> 225  (240)     0.22
//   200 of 16..64      46.3 -> 25.5 (32.0)    0.29
//   150 of 16..32      25.0 -> 11.1 (15.2)    0.44
//   400 of 16..64      61.3 -> 50.7 (71.4)    0.53
//   300 of 16..24      21.0 -> 20.6 (24.7)    1.09
// And the batched kernel has to take longer than the host does here: at least
// its longest system by itself, at 10 us per iteration and 4.3 for every tile
// after the first, against 300 us and 35 for each system (87 for a mixed one,
// whose reliable updates are steps of the host).  Iterations: 5.5 sqrt(n), of a
// mixed system with two threads per row and more (normal equations, whose
// condition is a square) 12 sqrt(n).  Whole call, ms:
//   1 fairing of 8 x 8 vertices      0.57 -> 0.37    5 of 10 x 9           0.81 -> 0.65
//   20 fairing of 10 x 10            1.29 -> 1.48    20 x 20               3.39 -> 1.81
//   20 fairing of 10 x 10, mixed     1.49 -> 2.51    20 x 20               3.78 -> 2.66
//   60 LSCM of 12 x 12, mixed        5.42 -> 6.96    16 x 16               9.60 -> 7.89
//   60 fairing of 20 x 20, mixed     5.08 -> 7.03    in FP64               4.92 -> 4.17
bool persist_batch_pays(const std::vector<SysView>& views) {
  const int n_sm = sm_count();
  double longest = 0.0, batched = 0.0, host = 300.0;
  for (const SysView& v : views) {
    longest = std::max(longest, persist_time(v, n_sm));
    const double iteration = std::min(70.0, 10.0 + 4.3 * (double)(v.n_tiles - 1));
    const bool mixed = v.r32 != nullptr;
    batched = std::max(batched, (mixed && v.tpr >= 2 ? 12.0 : 5.5) * std::sqrt((double)v.n) * (v.df ? 0.78 : 1.0) * iteration);
    host += mixed ? 87.0 : 35.0;
  }
  return (double)views.size() <= kPersistBatchRatio * longest && host <= batched;
}

cudaError_t persist_batch(std::vector<PersistSystem>& systems, cudaStream_t s, float* ms, bool* ran) {
  *ran = false;
  struct Lane {
    cudaStream_t s = nullptr;
    int sys = -1, sms = 0;
    unsigned int seq0 = 0;
    double t_due = 0.0;          // us (now_us)
    long long iter0 = 0;
  };
  using Clock = std::chrono::steady_clock;
  const Clock::time_point t_begin = Clock::now();
  auto now_us = [&]() { return std::chrono::duration<double, std::micro>(Clock::now() - t_begin).count(); };
  const int n = (int)systems.size(), n_sm = sm_count();
  std::vector<Lane> lanes((size_t)std::min(n, kPersistLanes));
  std::vector<std::unique_ptr<ViewGraph>> graphs;
  std::vector<size_t> at((size_t)n + 1, 0);
  ChunkMirror* mirrors = nullptr;
  char* exch = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaError_t e = cudaSuccess;
  auto ok = [&](cudaError_t r) {
    if (e == cudaSuccess) e = r;
    return e == cudaSuccess;
  };
  for (int i = 0; i < n; ++i)
    at[(size_t)i + 1] = at[(size_t)i] + align256(persist_bytes(systems[i].view.n, systems[i].view.n_tiles));
  ok(cudaHostAlloc((void**)&mirrors, sizeof(ChunkMirror) * (size_t)n, cudaHostAllocMapped));
  ok(cudaMallocAsync((void**)&exch, at[(size_t)n], s));
  if (ok(e)) ok(cudaMemsetAsync(exch, 0, at[(size_t)n], s));
  ok(cudaEventCreate(&e0));
  ok(cudaEventCreate(&e1));
  if (ok(e)) ok(cudaEventRecord(e0, s));
  for (Lane& l : lanes) {
    if (ok(e)) ok(cudaStreamCreateWithFlags(&l.s, cudaStreamNonBlocking));
    if (ok(e)) ok(cudaStreamWaitEvent(l.s, e0, 0));
  }
  if (ok(e)) std::memset((void*)mirrors, 0, sizeof(ChunkMirror) * (size_t)n);
  std::vector<int> order((size_t)n);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return persist_time(systems[a].view, n_sm) > persist_time(systems[b].view, n_sm);
  });
  // with room for all at once the clusters go first: spread CTAs of the grids
  // would leave no GPC with enough free SMs
  int all = 0;
  for (const PersistSystem& p : systems) all += p.plan[p.mixed ? 1 : 0].grid;
  if (all <= n_sm)
    std::stable_partition(order.begin(), order.end(),
                          [&](int i) { return systems[i].plan[systems[i].mixed ? 1 : 0].cluster; });
  for (int i = 0; i < n && ok(e); ++i) {
    graphs.emplace_back(new ViewGraph());
    graphs.back()->persist_bind(systems[i].layout, systems[i].plan, exch + at[(size_t)i]);
    graphs.back()->persist(true);
  }
  std::vector<int> waiting(order);     // longest first
  std::vector<char> fp64((size_t)n, 0);
  std::vector<double> us_per_iter((size_t)n, 0.0);
  int left = n, sms_busy = 0;
  auto seq_of = [&](int i) { return __atomic_load_n(&mirrors[i].seq, __ATOMIC_ACQUIRE); };
  auto start = [&](Lane& l) {
    const int i = l.sys;
    const bool mixed = systems[i].mixed && !fp64[(size_t)i];
    *ran = true;
    mirrors[i].budget = kPersistBatchIters;
    l.iter0 = mirrors[i].st.iter;
    l.t_due = now_us() + chunk_due_us(mixed, kPersistBatchIters, us_per_iter[(size_t)i]);
    l.seq0 = seq_of(i);
    if (ok(graphs[(size_t)i]->prepare(systems[i].view, mixed, &mirrors[i], l.s))) ok(graphs[(size_t)i]->launch(l.s));
  };
  while (left > 0 && ok(e)) {
    bool idle = true;
    for (Lane& l : lanes) {
      if (l.sys >= 0) {
        if (seq_of(l.sys) == l.seq0) {
          if (!ok(graphs[(size_t)l.sys]->advance(l.s))) break;
          continue;
        }
        idle = false;
        const int i = l.sys;
        const SysState& h = mirrors[i].st;
        if (h.iter > l.iter0)
          us_per_iter[(size_t)i] = (double)mirrors[i].t_ns * 1e-3 / (double)(h.iter - l.iter0);
        if (h.status == ST_STAGNATION && !h.fell_back && h.precision == 1) {
          // FP32 cannot track this system: it continues in FP64 from its x
          fp64[(size_t)i] = 1;
          mirrors[i].st.stage = 0;
          if (ok(chunk_fallback_fp64(systems[i].view.st, l.s))) start(l);
          continue;
        }
        if (h.stage != 3) {
          start(l);
          continue;
        }
        systems[i].state = h;
        if (h.status == ST_DEVICE_ERR) {
          set_error("batched solve: a wait of the persistent kernel timed out");
          ok(cudaErrorLaunchTimeout);
        }
        sms_busy -= l.sms;
        l.sys = -1;
        --left;
      }
      for (size_t q = 0; q < waiting.size() && ok(e); ++q) {
        const int c = graphs[(size_t)waiting[q]]->persist_ctas(systems[waiting[q]].mixed);
        if (sms_busy > 0 && sms_busy + c > n_sm) continue;
        l.sys = waiting[q];
        l.sms = c;
        sms_busy += c;
        waiting.erase(waiting.begin() + (long)q);
        start(l);
        idle = false;
        break;
      }
    }
    if (idle) {
      double due = 1e9;
      for (const Lane& l : lanes)
        if (l.sys >= 0) due = std::min(due, l.t_due);
      poll_pause(due - now_us());
    }
  }
  for (Lane& l : lanes) {
    if (!l.s) continue;
    const cudaError_t r = cudaStreamSynchronize(l.s);
    ok(r);
    cudaStreamDestroy(l.s);
  }
  if (e1 && ok(e) && ok(cudaEventRecord(e1, s)) && ok(cudaEventSynchronize(e1))) {
    float t = 0.f;
    cudaEventElapsedTime(&t, e0, e1);
    if (ms) *ms = t;
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (exch) cudaFreeAsync(exch, s);
  if (mirrors) cudaFreeHost(mirrors);
  return e;
}

// ---------------------------------------------------------------------------
// Per-system device slot.
// ---------------------------------------------------------------------------
size_t SystemSlot::bytes_for(int n, int tile_rows, bool mixed) {
  const size_t n8 = align256((size_t)std::max(2, n + 2) * sizeof(double));
  const size_t n4 = align256((size_t)std::max(4, n + 4) * sizeof(float));
  const int n_tiles = std::max(1, (n + tile_rows - 1) / tile_rows);
  const size_t parts = align256((size_t)n_tiles * kParts * sizeof(double));
  const size_t st = align256(sizeof(SysState));
  // mixed systems also carry the FP64 r, p, q of a possible FP64 fallback
  return mixed ? (5 * n8 + 4 * n4 + parts + st) : (5 * n8 + parts + st);
}

cudaError_t SystemSlot::alloc(DeviceCRS* Am, bool mx, cudaStream_t s, bool dfl) {
  A = Am;
  mixed = mx;
  df = dfl && !mx && Am->vadf != nullptr && Am->dinvdf != nullptr;
  const int n = A->n;
  bytes = bytes_for(n, A->tile_rows, mixed);
  NLGB_CUDA_TRY(cudaMallocAsync(&block, bytes, s));
  char* p = static_cast<char*>(block);
  const size_t n8 = align256((size_t)std::max(2, n + 2) * sizeof(double));
  const size_t n4 = align256((size_t)std::max(4, n + 4) * sizeof(float));
  std::memset(&view, 0, sizeof(view));
  view.n = n;
  view.tile_rows = A->tile_rows;
  view.n_tiles = std::max(1, (n + A->tile_rows - 1) / A->tile_rows);
  view.tpr = A->tpr;
  view.rp = A->rp; view.ci = A->ci; view.va = A->va; view.va32 = A->va32;
  view.dinv = A->dinv; view.dinv32 = A->dinv32;
  if (df) {
    view.df = 1;
    view.vadf = A->vadf;
    view.dinvdf = A->dinvdf;
  }
  view.b = reinterpret_cast<double*>(p); p += n8;
  view.x = reinterpret_cast<double*>(p); p += n8;
  view.r = reinterpret_cast<double*>(p); p += n8;
  view.p = reinterpret_cast<double*>(p); p += n8;
  view.q = reinterpret_cast<double*>(p); p += n8;
  if (mixed) {
    view.r32 = reinterpret_cast<float*>(p); p += n4;
    view.p32 = reinterpret_cast<float*>(p); p += n4;
    view.q32 = reinterpret_cast<float*>(p); p += n4;
    view.c32 = reinterpret_cast<float*>(p); p += n4;
  }
  view.part = reinterpret_cast<double*>(p);
  p += align256((size_t)view.n_tiles * kParts * sizeof(double));
  view.st = reinterpret_cast<SysState*>(p);
  return cudaSuccess;
}

cudaError_t SystemSlot::start(const double* b, const double* x0, const SolveParams& prm,
                              cudaStream_t s) {
  const size_t n = (size_t)view.n;
  NLGB_CUDA_TRY(cudaMemcpyAsync(const_cast<double*>(view.b), b, n * sizeof(double), cudaMemcpyDefault, s));
  if (x0) NLGB_CUDA_TRY(cudaMemcpyAsync(view.x, x0, n * sizeof(double), cudaMemcpyDefault, s));
  else NLGB_CUDA_TRY(cudaMemsetAsync(view.x, 0, n * sizeof(double), s));   // 0.0 in either form
  if (df && x0) NLGB_CUDA_TRY(df_pack(view.x, (long long)n, s));
  if (mixed) {
    NLGB_CUDA_TRY(cudaMemsetAsync(view.p32, 0, n * sizeof(float), s));
    NLGB_CUDA_TRY(cudaMemsetAsync(view.c32, 0, n * sizeof(float), s));
  }
  SysState h;
  std::memset(&h, 0, sizeof(h));
  const long long max_iter = prm.max_iter >= 0 ? prm.max_iter : 5LL * view.n;
  h.thresh2 = prm.eps * prm.eps;
  h.max_iter = max_iter;
  h.status = ST_RUNNING;
  h.max_outer = std::max(1, prm.max_outer);
  h.in_thresh2 = prm.inner_eps * prm.inner_eps;
  h.in_max = (int)std::max(1LL, std::min<long long>(max_iter, 1000));
  h.precision = mixed ? 1 : 0;
  h.stage = 0;
  // cudaMemcpyAsync from pageable memory is staged synchronously, so the
  // stack copy may go out of scope after the call.
  NLGB_CUDA_TRY(cudaMemcpyAsync(view.st, &h, sizeof(h), cudaMemcpyHostToDevice, s));
  return cudaSuccess;
}

void SystemSlot::release(cudaStream_t s) {
  if (block) cudaFreeAsync(block, s);
  block = nullptr;
}

}  // namespace nlgb
