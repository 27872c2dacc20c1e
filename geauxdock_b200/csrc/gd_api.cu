// gd_api.cu -- the C ABI of libgdock.so: resident ensembles, the drop-in
// Dock family, and pose evaluation.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <ctime>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

#include "gd_pack.h"

using namespace gd;

namespace {

struct Options {
  int kernel = GD_KERNEL_BATCHED;
  int precision = GD_PREC_FP32_KAHAN;  // FP32 pair terms, compensated reductions
  int warps = 0;  // 0: choose from occupancy
  int kpl = 0;    // pair-tile shape, 0: default_pair_tile
  int ab = 0;
  int graph = 1;  // replay whole exchange intervals from a captured graph
  int stage = -1; // protein conformation in shared memory: 1 staged, 0 through L1, -1 chosen
  int eval_cache = 1;  // gd_eval_poses keeps its device block and stream for the next call
  int dock_cache = 1;  // Dock keeps its device state per GPU between calls
  int dock_device_pack = 1;  // Dock refills that state on the GPU from the Complex CopyH2D put there
  int dock_record_direct = 1;  // Dock's kernels write Records straight into a GPU-mapped host array
  int replica_warps = 1;     // order of the energy sums: 1 the one-warp kernel's, 2, 4 or 8 that of a replica split over so many
  int device_base = 0;        // the drop-in API's GPU g is CUDA device device_base + g
  long long wait_limit = 0;   // microseconds of a bounded shared-memory wait (0: one second)
  int stall_test = 0;         // test hook: staging (1) or cluster (2) barriers that never complete (bounded waits run out)
};
Options g_opt;
int g_ngpu = -1;
std::mutex g_mu;

int ngpu()
{
  std::lock_guard<std::mutex> lk(g_mu);
  if (g_ngpu < 0) {
    const char *e = std::getenv("GDOCK_NGPU");
    g_ngpu = e ? std::max(1, std::atoi(e)) : 1;
  }
  return g_ngpu;
}

Options opts()
{
  std::lock_guard<std::mutex> lk(g_mu);
  return g_opt;
}

// Field by field: Options has padding, whose bytes a copy need not keep.
bool same_options(const Options &a, const Options &b)
{
  return a.kernel == b.kernel && a.precision == b.precision && a.warps == b.warps && a.kpl == b.kpl &&
         a.ab == b.ab && a.graph == b.graph && a.stage == b.stage && a.dock_cache == b.dock_cache &&
         a.dock_device_pack == b.dock_device_pack && a.replica_warps == b.replica_warps &&
         a.device_base == b.device_base && a.wait_limit == b.wait_limit && a.stall_test == b.stall_test;
}

}  // namespace

struct gd_ensemble;

struct gd_rng {
  uint64_t seed = 0;
  uint64_t calls = 0;
  int seeded = 0;
  uint64_t dock_calls = 0;   // Dock calls on this handle's GPU
  uint64_t dock_reused = 0;  // of them, refills of the kept device state
  // Dock's resident state on this handle's GPU, kept between calls and refilled
  // in place when the next Complex has the same shapes
  gd_ensemble *dock = nullptr;
  std::vector<unsigned char> dock_prt;  // protein bytes the cached pocket was packed from
  Options dock_opt;                     // options the cached ensemble was configured with
};

struct gd_ensemble {
  int device = 0;
  cudaStream_t st = nullptr;
  std::vector<DevPocket> pockets;
  std::vector<DevJobBuf> jobs;
  std::vector<std::vector<int>> rep_prt;  // per job, per replica: protein conformation
  DevJob *d_jobs = nullptr;
  WorkItem *d_items = nullptr;
  int n_items = 0;
  std::vector<WorkItem> h_items;   // host copy of d_items (the autotuner samples it)
  int *d_queue = nullptr;
  int *d_err = nullptr;
  int kernel = GD_KERNEL_BATCHED;
  int precision = GD_PREC_FP32;
  TileConfig tc{8, 1, 8};
  int grid = 0;
  size_t smem = 0;
  int Pmax = 0, lig_slots = 0;
  int step = 0;
  // replica exchange over all jobs: pair-count prefix sums per parity
  int *d_xoff = nullptr;
  int xtot = 0;
  // device copy of the step counter and the captured exchange interval
  int *d_step = nullptr;
  cudaGraphExec_t gexec = nullptr;
  int g_chunk = 0;
  bool use_graph = true;
  // timing of the Monte Carlo launches
  std::vector<cudaEvent_t> ev;
  int ev_used = 0;
  uint32_t wait_limit = 0, stall_bytes = 0;  // bounded-wait limit and the test hooks (options)
  bool stall_nodes = false;
  int launches = 0;      // Monte Carlo kernel launches (or graph replays of one)
  int all_launches = 0;  // every kernel of this library launched on the stream
  // pose evaluation's blocks (EvalBlock)
  unsigned char *eval_dev = nullptr;
  std::unique_ptr<unsigned char[]> eval_host;
  size_t eval_bytes = 0;
};
constexpr size_t kEvalKeep = 32u << 20;

namespace {

int set_device(int d) { GD_CUDA(cudaSetDevice(d)); return GD_OK; }

// CUDA device of the drop-in API's GPU g.
int dev_of(int g) { return opts().device_base + g; }

// Work items: runs of consecutive replicas of one job with the same protein
// conformation, at most `warps` long; heaviest (L x P) first.
int build_items(gd_ensemble *e)
{
  std::vector<WorkItem> items;
  std::vector<double> cost;
  const int R = e->tc.warps_per_cta / std::max(1, e->tc.group);  // replicas per CTA
  for (int j = 0; j < (int)e->jobs.size(); ++j) {
    const std::vector<int> &pr = e->rep_prt[j];
    const double c = (double)e->jobs[j].dj.natom * e->jobs[j].dj.npoint_pad;
    int r = 0;
    const int n = (int)pr.size();
    while (r < n) {
      int k = 1;
      while (r + k < n && k < R && pr[r + k] == pr[r]) ++k;
      items.push_back(WorkItem{j, pr[r], r, k});
      cost.push_back(c);
      r += k;
    }
  }
  std::vector<int> ord(items.size());
  std::iota(ord.begin(), ord.end(), 0);
  std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return cost[a] > cost[b]; });
  std::vector<WorkItem> sorted(items.size());
  for (size_t i = 0; i < ord.size(); ++i) sorted[i] = items[ord[i]];
  if (e->d_items) cudaFree(e->d_items);
  e->d_items = nullptr;
  e->n_items = (int)sorted.size();
  e->h_items = sorted;
  if (!sorted.empty()) {
    GD_CUDA(cudaMalloc(&e->d_items, sizeof(WorkItem) * sorted.size()));
    GD_CUDA(cudaMemcpy(e->d_items, sorted.data(), sizeof(WorkItem) * sorted.size(), cudaMemcpyHostToDevice));
  }
  return GD_OK;
}

size_t smem_for(const gd_ensemble *e, const TileConfig &tc)
{
  return kernel_smem_bytes(tc.stage ? e->Pmax : 0, e->Pmax, e->lig_slots, e->precision, tc);
}

// Check a tile shape, fix its staging, work items and grid.
int configure(gd_ensemble *e, TileConfig tc)
{
  if (e->kernel == GD_KERNEL_PLAIN) tc.group = 1;
  if (tc.group != 1 && tc.group != 2 && tc.group != 4 && tc.group != 8 && tc.group != 16)
    return fail(GD_E_INVALID, "warps per replica = %d (1, 2, 4, 8 or 16)", tc.group);
  if (tc.warps_per_cta < 1 || tc.warps_per_cta * 32 > kMaxCtaThreads || tc.warps_per_cta % tc.group)
    return fail(GD_E_INVALID, "warps per CTA = %d outside [1, %d] or not a multiple of the %d warps per replica",
                tc.warps_per_cta, kMaxCtaThreads / 32, tc.group);
  // a pocket too large to stage is read through L1
  if (tc.stage && smem_for(e, tc) > kSmemLimit) tc.stage = 0;
  const size_t smem = smem_for(e, tc);
  if (smem > kSmemLimit)
    return fail(GD_E_CAPACITY, "%d warps per CTA need %zu B of shared memory (limit %zu)", tc.warps_per_cta, smem,
                kSmemLimit);
  const int occ = kernel_occupancy(0, e->precision, tc, smem);
  if (occ < 1) return fail(GD_E_INVALID, "tile (warps %d, kpl %d, ab %d) cannot launch", tc.warps_per_cta, tc.kpl, tc.ab);
  int nsm = 0;
  GD_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, e->device));
  e->tc = tc;
  e->smem = smem;
  if (e->gexec) {
    cudaGraphExecDestroy(e->gexec);
    e->gexec = nullptr;
  }
  GD_TRY(build_items(e));
  e->grid = std::max(1, std::min(e->n_items, occ * nsm));
  return GD_OK;
}

// Work items of R replicas at most (build_items).
long long count_items(const std::vector<int> &pr, int R)
{
  long long items = 0;
  for (size_t r = 0, k; r < pr.size(); r += k) {
    for (k = 1; r + k < pr.size() && (int)k < R && pr[r + k] == pr[r]; ++k) {}
    ++items;
  }
  return items;
}
long long count_items(const gd_ensemble *e, int R)
{
  long long items = 0;
  for (const std::vector<int> &pr : e->rep_prt) items += count_items(pr, R);
  return items;
}

ShapeQuery shape_query(const gd_ensemble *e, int stage_opt, int nsm)
{
  ShapeQuery q;
  q.precision = e->precision;
  q.Pmax = e->Pmax;
  q.lig_slots = e->lig_slots;
  q.nsm = nsm;
  q.stage_opt = stage_opt;
  q.items = [e](int R) { return count_items(e, R); };
  q.loads = [e](int R, std::vector<std::pair<double, long long>> &out) {
    for (size_t j = 0; j < e->jobs.size(); ++j)
      out.emplace_back((double)e->jobs[j].dj.natom * e->jobs[j].dj.npoint_pad, count_items(e->rep_prt[j], R));
  };
  return q;
}

// Warps per replica and replicas per CTA from occupancy: a team each where one
// wave holds them, else base.group warps each, fewest waves of work items, then
// most resident warps per SM.
// stage_opt: -1 chooses between staging the pocket and reading it through L1.
int choose_warps(gd_ensemble *e, TileConfig base, int stage_opt = -1)
{
  int nsm = 0;
  GD_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, e->device));
  int grid = 0;
  const ShapeQuery q = shape_query(e, stage_opt, nsm);
  if ((e->kernel == GD_KERNEL_BATCHED && choose_team(q, base, grid)) || (base.group == 1 && choose_spread(q, base, grid))) {
    if (e->kernel == GD_KERNEL_BATCHED) choose_waves(q, base, grid);
    return configure(e, base);
  }
  double best = 1e300;
  const int G = e->kernel == GD_KERNEL_PLAIN ? 1 : std::max(1, base.group);
  int best_w = std::max(8, G), best_stage = 1;
  for (int stage = 1; stage >= 0; --stage)
  for (int w = std::max(2, G); w <= kMaxCtaThreads / 32; w += (w < G ? 1 : G)) {
    if (stage_opt >= 0 && stage != stage_opt) continue;
    if (w % G) continue;
    TileConfig tc = base;
    tc.warps_per_cta = w;
    tc.stage = stage;
    tc.group = G;
    const size_t smem = smem_for(e, tc);
    if (smem > kSmemLimit) continue;
    const int occ = kernel_occupancy(0, e->precision, tc, smem);
    if (occ < 1) continue;
    // items and the slowest SM's load (items are equal-cost within a job)
    const long long items = count_items(e, w / G);
    const long long slots = (long long)occ * nsm;
    const long long waves = (items + slots - 1) / slots;
    // time ~ waves * (warps resident per SM); fewer resident warps per SM than 16 also hurts latency hiding
    const int resident = occ * w;
    double t = (double)waves * std::max(resident, 16) / (double)std::min(resident, 32);
    if (!stage) t *= 1.05;  // L1 reads of the pocket: prefer staging when occupancy is equal
    // of equal shapes up to 8 warps the largest: each CTA has its own pair tables, which L1 loses
    // (3520 replicas, 24 warps per SM as 6 CTAs of 4 warps: 3.10 ms for 10 steps, as 3 of 8: 2.96 ms);
    // above, smaller items balance uneven ligands better (32 ligands x 400 replicas, 4 steps, 12 warps
    // 5.60 ms, 8 warps 5.32 ms)
    if (w <= 8 ? t < best + 1e-9 : t < best - 1e-9) {
      best = t;
      best_w = w;
      best_stage = stage;
    }
  }
  TileConfig tc = base;
  tc.warps_per_cta = best_w;
  tc.stage = best_stage;
  tc.group = G;
  if (e->kernel == GD_KERNEL_BATCHED && smem_for(e, tc) <= kSmemLimit) {
    grid = (int)std::min(count_items(e, best_w / G), (long long)kernel_occupancy(0, e->precision, tc, smem_for(e, tc)) * nsm);
    choose_waves(q, tc, grid);
  }
  return configure(e, tc);
}

int upload_jobs(gd_ensemble *e)
{
  std::vector<DevJob> h(e->jobs.size());
  for (size_t j = 0; j < e->jobs.size(); ++j) h[j] = e->jobs[j].dj;
  if (e->d_jobs) cudaFree(e->d_jobs);
  GD_CUDA(cudaMalloc(&e->d_jobs, sizeof(DevJob) * std::max<size_t>(h.size(), 1)));
  GD_CUDA(cudaMemcpy(e->d_jobs, h.data(), sizeof(DevJob) * h.size(), cudaMemcpyHostToDevice));
  return GD_OK;
}

int finish_create(gd_ensemble *e)
{
  e->Pmax = 0;
  int Lmax = 1;
  e->rep_prt.resize(e->jobs.size());
  for (size_t j = 0; j < e->jobs.size(); ++j) {
    const DevJob &J = e->jobs[j].dj;
    e->Pmax = std::max(e->Pmax, J.npoint_pad);
    Lmax = std::max(Lmax, J.natom);
  }
  e->lig_slots = (Lmax + 3) & ~3;
  GD_TRY(upload_jobs(e));
  {
    const size_t nj = e->jobs.size();
    std::vector<int> xoff(2 * (nj + 1), 0);
    for (int par = 0; par < 2; ++par)
      for (size_t j = 0; j < nj; ++j) {
        const DevJob &J = e->jobs[j].dj;
        const int np = J.ntmp >= 2 ? (J.ntmp - par) / 2 : 0;
        xoff[par * (nj + 1) + j + 1] = xoff[par * (nj + 1) + j] + J.nprt * J.nlig * np;
      }
    e->xtot = std::max(xoff[nj], xoff[2 * (nj + 1) - 1]);
    GD_CUDA(cudaMalloc(&e->d_xoff, sizeof(int) * xoff.size()));
    GD_CUDA(cudaMemcpy(e->d_xoff, xoff.data(), sizeof(int) * xoff.size(), cudaMemcpyHostToDevice));
  }
  GD_CUDA(cudaMalloc(&e->d_step, sizeof(int)));
  GD_CUDA(cudaMalloc(&e->d_queue, sizeof(int)));
  // error words: [0] kernel flags (kErr*), [1..3] the device packer's failure details
  GD_CUDA(cudaMalloc(&e->d_err, 4 * sizeof(int)));
  GD_CUDA(cudaMemset(e->d_err, 0, 4 * sizeof(int)));
  GD_CUDA(cudaStreamCreateWithFlags(&e->st, cudaStreamNonBlocking));
  const Options o = opts();
  e->kernel = o.kernel;
  e->precision = o.precision;
  e->use_graph = o.graph != 0;
  e->wait_limit = (uint32_t)o.wait_limit;
  e->stall_bytes = o.stall_test == 1 ? 16u : 0u;
  e->stall_nodes = o.stall_test == 2;
  TileConfig tc{o.warps > 0 ? o.warps : 8, o.kpl, o.ab, o.stage != 0 ? 1 : 0, o.replica_warps};
  default_pair_tile(tc.kpl, tc.ab);
  if (e->precision == GD_PREC_FP64) tc.kpl = 1, tc.ab = 8, tc.group = 1;
  // replica_warps > 1 names the order the sums are combined in; FP64 and the plain kernel have one
  if (e->kernel == GD_KERNEL_BATCHED) tc.split = tc.group;
  if (o.warps > 0) return configure(e, tc);
  return choose_warps(e, tc, o.stage);
}

int read_replica_prt(gd_ensemble *e, size_t j, const std::vector<ReplicaMC> &reps)
{
  e->rep_prt[j].resize(reps.size());
  for (size_t r = 0; r < reps.size(); ++r) e->rep_prt[j][r] = reps[r].idx_prt;
  return GD_OK;
}

cudaEvent_t next_event(gd_ensemble *e)
{
  if (e->ev_used == (int)e->ev.size()) {
    cudaEvent_t x;
    if (cudaEventCreate(&x) != cudaSuccess) return nullptr;
    e->ev.push_back(x);
  }
  return e->ev[e->ev_used++];
}

int check_err(gd_ensemble *e)
{
  int h[4] = {0, 0, 0, 0};
  GD_CUDA(cudaMemcpy(h, e->d_err, sizeof(h), cudaMemcpyDeviceToHost));
  if (h[0] & kErrPack) {
    if (h[1] == kPackFailShape)
      return fail(GD_E_INVALID, "the Complex on the GPU differs in %s (%d) from the one the host described",
                  pack_field_name(h[2]), h[3]);
    return fail(h[1] == kPackFailCapacity ? GD_E_CAPACITY : GD_E_INVALID, "invalid Complex: %s: %d",
                pack_field_name(h[2]), h[3]);
  }
  if (h[0] & kErrTimeout) return fail(GD_E_TIMEOUT, "a bounded wait for a shared-memory bulk copy gave up");
  return GD_OK;
}

KArgs mc_args(gd_ensemble *e, int s_begin, int nsteps, int flags, const int *d_step);

int launch_mc(gd_ensemble *e, int s_begin, int nsteps, int flags)
{
  cudaEvent_t e0 = next_event(e), e1 = next_event(e);
  if (!e0 || !e1) return fail(GD_E_CUDA, "cudaEventCreate failed");
  GD_CUDA(cudaEventRecord(e0, e->st));
  if (e->kernel == GD_KERNEL_PLAIN) {
    for (size_t j = 0; j < e->jobs.size(); ++j)
      GD_CUDA(launch_plain(e->d_jobs + j, e->jobs[j].dj.nrep, s_begin, nsteps, flags, e->d_err, e->st));
    e->launches += (int)e->jobs.size();
    e->all_launches += (int)e->jobs.size();
  } else {
    GD_CUDA(cudaMemsetAsync(e->d_queue, 0, sizeof(int), e->st));
    GD_CUDA(launch_kernel(0, e->precision, e->tc, mc_args(e, s_begin, nsteps, flags, nullptr), e->grid, e->st));
    e->launches += 1;
    e->all_launches += 1;
  }
  GD_CUDA(cudaEventRecord(e1, e->st));
  return GD_OK;
}

KArgs mc_args(gd_ensemble *e, int s_begin, int nsteps, int flags, const int *d_step)
{
  KArgs a{};
  a.jobs = e->d_jobs;
  a.items = e->d_items;
  a.n_items = e->n_items;
  a.queue = e->d_queue;
  a.err = e->d_err;
  a.s_begin = s_begin;
  a.nsteps = nsteps;
  a.flags = flags | (e->stall_nodes ? kMcStallNodes : 0);
  a.d_step = d_step;
  a.P = e->tc.stage ? e->Pmax : 0;
  a.Pall = e->Pmax;
  a.lig_slots = e->lig_slots;
  a.wait_limit = e->wait_limit;
  a.stall_bytes = (uint16_t)e->stall_bytes;
  return a;
}

// One exchange interval (queue reset, Monte Carlo chunk of `chunk` steps from
// *d_step, exchange sweep, *d_step += chunk) captured once and replayed.
int interval_graph(gd_ensemble *e, int chunk)
{
  if (e->gexec && e->g_chunk == chunk) return GD_OK;
  if (e->gexec) {
    cudaGraphExecDestroy(e->gexec);
    e->gexec = nullptr;
  }
  cudaGraph_t g = nullptr;
  GD_CUDA(cudaStreamBeginCapture(e->st, cudaStreamCaptureModeThreadLocal));
  cudaError_t ce = cudaMemsetAsync(e->d_queue, 0, sizeof(int), e->st);
  if (ce == cudaSuccess) ce = launch_kernel(0, e->precision, e->tc, mc_args(e, 0, chunk, kMcStoreAccept, e->d_step), e->grid, e->st);
  if (ce == cudaSuccess)
    ce = launch_exchange_all(e->d_jobs, e->d_xoff, (int)e->jobs.size(), e->xtot, 0, e->d_step, chunk, chunk, e->st);
  if (ce == cudaSuccess) ce = launch_advance_step(e->d_step, chunk, e->st);
  const cudaError_t ee = cudaStreamEndCapture(e->st, &g);
  if (ce != cudaSuccess || ee != cudaSuccess) {
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    return fail(GD_E_CUDA, "graph capture: %s", cudaGetErrorString(ce != cudaSuccess ? ce : ee));
  }
  ce = cudaGraphInstantiate(&e->gexec, g, 0);
  cudaGraphDestroy(g);
  if (ce != cudaSuccess) return fail(GD_E_CUDA, "cudaGraphInstantiate: %s", cudaGetErrorString(ce));
  e->g_chunk = chunk;
  return GD_OK;
}

int exchange_sweep(gd_ensemble *e, int x)
{
  if (e->xtot <= 0) return GD_OK;
  GD_CUDA(launch_exchange_all(e->d_jobs, e->d_xoff, (int)e->jobs.size(), e->xtot, x, nullptr, 0, 0, e->st));
  e->all_launches += 1;
  return GD_OK;
}

// nsteps steps from e->step, cut at exchange boundaries.  Whole exchange
// intervals of a plain run (no records) replay the captured interval graph.
int advance(gd_ensemble *e, int nsteps, int spx, int f_first, int f_all, int f_last)
{
  int done = 0;
  if (e->use_graph && e->kernel == GD_KERNEL_BATCHED && spx > 0 && f_first == 0 && f_all == 0 &&
      f_last == kMcStoreAccept && e->step % spx == 0 && nsteps >= spx) {
    const int n_int = nsteps / spx;
    if (interval_graph(e, spx) == GD_OK) {
      // a kernel argument rather than a copy from pageable memory, which
      // could wait for the stream
      GD_CUDA(launch_set_step(e->d_step, e->step, e->st));
      cudaEvent_t e0 = next_event(e), e1 = next_event(e);
      if (!e0 || !e1) return fail(GD_E_CUDA, "cudaEventCreate failed");
      GD_CUDA(cudaEventRecord(e0, e->st));
      for (int k = 0; k < n_int; ++k) GD_CUDA(cudaGraphLaunch(e->gexec, e->st));
      GD_CUDA(cudaEventRecord(e1, e->st));
      e->launches += n_int;
      e->all_launches += 1 + 3 * n_int;
      e->step += n_int * spx;
      done = n_int * spx;
    } else {
      e->use_graph = false;   // capture unavailable: launch chunk by chunk
    }
  }
  while (done < nsteps) {
    int chunk = nsteps - done;
    if (spx > 0) chunk = std::min(chunk, spx - (e->step % spx));
    const int f = f_all | (done == 0 ? f_first : 0) | (done + chunk == nsteps ? f_last : 0);
    GD_TRY(launch_mc(e, e->step, chunk, f));
    e->step += chunk;
    done += chunk;
    if (spx > 0 && e->step % spx == 0) GD_TRY(exchange_sweep(e, e->step / spx - 1));
  }
  return GD_OK;
}

void destroy(gd_ensemble *e)
{
  if (!e) return;
  cudaSetDevice(e->device);
  if (e->st) cudaStreamSynchronize(e->st);
  for (auto &j : e->jobs) free_job(j);
  for (auto &p : e->pockets) free_pocket(p);
  if (e->d_jobs) cudaFree(e->d_jobs);
  if (e->d_items) cudaFree(e->d_items);
  if (e->d_queue) cudaFree(e->d_queue);
  if (e->d_err) cudaFree(e->d_err);
  if (e->d_xoff) cudaFree(e->d_xoff);
  if (e->d_step) cudaFree(e->d_step);
  if (e->eval_dev) cudaFree(e->eval_dev);
  if (e->gexec) cudaGraphExecDestroy(e->gexec);
  for (auto x : e->ev) cudaEventDestroy(x);
  if (e->st) cudaStreamDestroy(e->st);
  delete e;
}

// Ensemble of one job from a Complex replica range (the Dock path).
int ensemble_from_complex_range(const Complex *c, int rb, int re, uint64_t seed, Record *rec, int device,
                                gd_ensemble **out)
{
  *out = nullptr;
  Tracer tr("create");
  GD_TRY(set_device(device));
  PocketData pk;
  JobData jd;
  GD_TRY(pocket_from_complex(c, pk));
  GD_TRY(job_from_complex(c, rb, re, seed, jd));
  jd.cell_room = true;  // Dock refills this state in place from later Complexes
  tr.mark("read Complex");
  gd_ensemble *e = new gd_ensemble;
  e->device = device;
  e->pockets.resize(1);
  e->jobs.resize(1);
  int rc = pack_pocket(pk, e->pockets[0]);
  tr.mark("pack pocket");
  if (rc == GD_OK) rc = pack_job(jd, e->pockets[0], c->enepara, rec != nullptr, rec, e->jobs[0]);
  tr.mark("pack job");
  if (rc == GD_OK) {
    e->rep_prt.resize(1);
    read_replica_prt(e, 0, jd.reps);
    rc = finish_create(e);
  }
  tr.mark("configure");
  if (rc != GD_OK) {
    destroy(e);
    return rc;
  }
  *out = e;
  return GD_OK;
}

// The shapes Dock's cached state was packed for, read from a host Complex
// without packing it: true if `c` (replicas [rb, re]) has exactly these.
bool same_dock_shapes(const gd_ensemble *e, const Complex *c, int rb, int re)
{
  if (e->jobs.size() != 1 || e->pockets.size() != 1) return false;
  const DevJob &J = e->jobs[0].dj;
  const ComplexSize &sz = c->size;
  if (sz.n_prt < 1 || sz.n_prt > GD_MAX_CONF_PRT || sz.n_lig < 1 || sz.n_lig > GD_MAX_CONF_LIG ||
      sz.kde_npoint < 0 || sz.kde_npoint > GD_MAXKDE || sz.n_rep > GD_MAX_REP || rb < 0 || re >= sz.n_rep || rb > re)
    return false;
  int P = 0;
  for (int i = 0; i < sz.n_prt; ++i) P = std::max(P, c->prt[i].prt_npoint);
  const int Ppad = ((P + kPointAlign - 1) / kPointAlign) * kPointAlign;
  int nk = 0;
  for (int k = 0; k < sz.kde_npoint; ++k) nk += c->kde.t[k] >= 0 && c->kde.t[k] < kLigTypes;
  if (J.natom != c->lig[0].lig_natom || J.nlig != sz.n_lig || J.nprt != sz.n_prt || J.ntmp != sz.n_tmp ||
      J.nmcs != sz.mcs_nrow || J.npoint_pad != Ppad || e->pockets[0].Ppad != Ppad || J.nkde != nk ||
      J.nrep != re - rb + 1 || J.rid_base != rb || J.nrep_total != sz.n_rep)
    return false;
  const std::vector<int> &prt = e->rep_prt[0];
  for (int r = rb; r <= re; ++r)
    if (c->replica[r].idx_prt != prt[r - rb]) return false;  // the work items group replicas by it
  return true;
}

// Refill of Dock's cached state on the GPU: the device packer reads the
// Complex that CopyH2D put at d_cx and writes the arenas the state already
// holds (no host packing, no copy of packed arrays).  A Complex the packer
// refuses sets the ensemble's error flag, which the kernels and check_err see.
int dock_refill_device(gd_ensemble *e, const Complex *d_cx, int rb, int re, int n_rep, uint64_t seed, Record *rec)
{
  const DevJob &J = e->jobs[0].dj;
  const DevPocket &pk = e->pockets[0];
  PackDst D{};
  D.job = e->d_jobs;
  D.par = const_cast<DevParams *>(J.par);
  D.ref4 = const_cast<float4 *>(J.ref4);
  D.err = e->d_err;
  D.lgrp = const_cast<int2 *>(J.lgrp);
  D.lcenter = const_cast<float *>(J.lcenter);
  D.pcenter = pk.center;
  D.tcc = const_cast<float *>(J.tcc);
  D.lig = const_cast<float4 *>(J.lig);
  D.kde = const_cast<float4 *>(J.kde);
  D.mcs = const_cast<float4 *>(J.mcs);
  D.pos = pk.pos;
  D.aux = pk.aux;
  D.ncdc = pk.ncdc;
  D.psp = const_cast<float *>(J.psp);
  D.pspmask = const_cast<uint32_t *>(J.pspmask);
  D.pcell = const_cast<int4 *>(J.pcell);
  D.pcell_cnt = const_cast<int *>(J.pcell_cnt);
  D.pcell_stride = J.pcell_stride;
  D.kslot = const_cast<int4 *>(J.kslot);
  D.kde_cap = std::max(J.nkde, 1);
  D.Ppad = pk.Ppad;
  D.nkde_expect = J.nkde;
  D.expect_L = J.natom;
  D.expect_nlig = J.nlig;
  D.expect_nprt = J.nprt;
  D.expect_M = J.nmcs;
  D.expect_ntmp = J.ntmp;
  D.rep = J.rep;
  D.run_acc = J.run_acc;
  D.stats = J.stats;
  D.minus_beta = const_cast<float *>(J.minus_beta);
  D.rec = rec;
  D.rep_begin = rb;
  D.nrep = re - rb + 1;
  D.nrep_total = n_rep;
  D.key0 = (uint32_t)seed;
  D.key1 = (uint32_t)(seed >> 32);
  GD_CUDA(cudaMemsetAsync(e->d_err, 0, 4 * sizeof(int), e->st));
  GD_CUDA(device_pack(d_cx, D, e->st));
  e->all_launches += 1;
  e->jobs[0].dj.key0 = D.key0;  // the host copy of the header follows the device one
  e->jobs[0].dj.key1 = D.key1;
  e->jobs[0].dj.rec = rec;
  return GD_OK;
}

// Dock's ensemble on GPU `device`: the handle's cached one refilled in place
// when the shapes are unchanged (no allocation and no reconfiguration), by the
// device packer from the Complex CopyH2D put on the GPU (d_cx; option
// dock_device_pack) or else by the host packer (the packed pocket kept when
// the protein bytes are unchanged); otherwise a new one, which the handle
// then keeps.
int dock_ensemble(gd_rng *h, const Complex *c, const Complex *d_cx, int rb, int re, uint64_t seed, Record *rec,
                  int device, gd_ensemble **out)
{
  *out = nullptr;
  const Options o = opts();
  const size_t prt_bytes = sizeof(Protein) * (size_t)std::max(0, std::min(c->size.n_prt, GD_MAX_CONF_PRT));
  gd_ensemble *e = h->dock;
  ++h->dock_calls;
  if (e && e->device == device && same_options(h->dock_opt, o) && o.dock_device_pack && d_cx &&
      same_dock_shapes(e, c, rb, re)) {
    Tracer tr("refill on the GPU");
    GD_TRY(set_device(device));
    GD_CUDA(cudaStreamSynchronize(e->st));
    e->step = 0;
    e->ev_used = 0;
    e->launches = 0;
    e->all_launches = 0;
    GD_TRY(dock_refill_device(e, d_cx, rb, re, c->size.n_rep, seed, rec));
    h->dock_prt.clear();  // the host packer's record of the packed protein no longer holds
    tr.mark("pack enqueued");
    ++h->dock_reused;
    *out = e;
    return GD_OK;
  }
  if (e && e->device == device && same_options(h->dock_opt, o) && e->jobs.size() == 1) {
    Tracer tr("refill");
    GD_TRY(set_device(device));
    GD_CUDA(cudaStreamSynchronize(e->st));
    JobData jd;
    GD_TRY(job_from_complex(c, rb, re, seed, jd));
    jd.cell_room = true;  // the arena keeps the size of the one it refills
    bool ok = true;
    const bool same_prt = h->dock_prt.size() == prt_bytes &&
                          std::memcmp(h->dock_prt.data(), c->prt, prt_bytes) == 0 &&
                          e->pockets[0].hdb_types == hdb_point_types(c->enepara);
    if (!same_prt) {
      PocketData pk;
      GD_TRY(pocket_from_complex(c, pk));
      DevPocket np;
      GD_TRY(pack_pocket(pk, np, &e->pockets[0], e->st));
      if (np.arena != e->pockets[0].arena) {
        free_pocket(np);
        ok = false;
      } else {
        e->pockets[0] = np;
        h->dock_prt.assign((const unsigned char *)c->prt, (const unsigned char *)c->prt + prt_bytes);
      }
    }
    tr.mark("pocket");
    if (ok) {
      DevJobBuf nj;
      GD_TRY(pack_job(jd, e->pockets[0], c->enepara, rec != nullptr, rec, nj, &e->jobs[0], e->st));
      const DevJob &A = e->jobs[0].dj, &B = nj.dj;
      if (nj.arena != e->jobs[0].arena) {
        free_job(nj);
        ok = false;
      } else {
        ok = A.natom == B.natom && A.nlig == B.nlig && A.nprt == B.nprt && A.ntmp == B.ntmp && A.nrep == B.nrep &&
             A.nkde == B.nkde && A.nmcs == B.nmcs && A.npoint_pad == B.npoint_pad;
        e->jobs[0] = nj;
        std::vector<int> prt_of(jd.reps.size());
        for (size_t r = 0; r < jd.reps.size(); ++r) prt_of[r] = jd.reps[r].idx_prt;
        ok = ok && prt_of == e->rep_prt[0];
      }
    }
    tr.mark("job");
    if (ok) {
      GD_CUDA(cudaMemcpyAsync(e->d_jobs, &e->jobs[0].dj, sizeof(DevJob), cudaMemcpyHostToDevice, e->st));
      GD_CUDA(cudaMemsetAsync(e->d_err, 0, sizeof(int), e->st));
      e->step = 0;
      e->ev_used = 0;
      e->launches = 0;
      e->all_launches = 0;
      ++h->dock_reused;
      *out = e;
      return GD_OK;
    }
    destroy(e);  // shapes changed: a new ensemble below
    h->dock = nullptr;
    h->dock_prt.clear();
  } else if (e) {
    destroy(e);
    h->dock = nullptr;
    h->dock_prt.clear();
  }
  GD_TRY(ensemble_from_complex_range(c, rb, re, seed, rec, device, &e));
  if (!o.dock_cache) {  // the caller destroys it after the call
    *out = e;
    return GD_OK;
  }
  h->dock = e;
  h->dock_prt.assign((const unsigned char *)c->prt, (const unsigned char *)c->prt + prt_bytes);
  h->dock_opt = o;
  *out = e;
  return GD_OK;
}

}  // namespace

void eval_drop_spaces();  // the blocks gd_eval_poses keeps

// =================================================================== C ABI
extern "C" {

int gd_set_ngpu(int n)
{
  if (n < 1) return fail(GD_E_INVALID, "ngpu = %d", n);
  std::lock_guard<std::mutex> lk(g_mu);
  g_ngpu = n;
  return GD_OK;
}

int gd_get_ngpu(void) { return ngpu(); }

int gd_set_option(const char *name, long long v)
{
  if (!name) return fail(GD_E_INVALID, "null option name");
  std::lock_guard<std::mutex> lk(g_mu);
  const std::string n(name);
  if (n == "kernel") {
    if (v != GD_KERNEL_BATCHED && v != GD_KERNEL_PLAIN) return fail(GD_E_INVALID, "kernel = %lld", v);
    g_opt.kernel = (int)v;
  } else if (n == "precision") {
    if (v < GD_PREC_FP32 || v > GD_PREC_FP64) return fail(GD_E_INVALID, "precision = %lld", v);
    g_opt.precision = (int)v;
  } else if (n == "warps") {
    if (v < 0 || v > kMaxCtaThreads / 32) return fail(GD_E_INVALID, "warps = %lld", v);
    g_opt.warps = (int)v;
  } else if (n == "kpl") {
    if (v != 0 && v != 1 && v != 2 && v != 4) return fail(GD_E_INVALID, "kpl = %lld", v);
    g_opt.kpl = (int)v;
  } else if (n == "ab") {
    if (v != 0 && v != 4 && v != 8) return fail(GD_E_INVALID, "ab = %lld", v);
    g_opt.ab = (int)v;
  } else if (n == "stage") {
    if (v < -1 || v > 1) return fail(GD_E_INVALID, "stage = %lld", v);
    g_opt.stage = (int)v;
  } else if (n == "dock_cache") {
    if (v != 0 && v != 1) return fail(GD_E_INVALID, "dock_cache = %lld", v);
    g_opt.dock_cache = (int)v;
  } else if (n == "eval_cache") {
    if (v != 0 && v != 1) return fail(GD_E_INVALID, "eval_cache = %lld", v);
    g_opt.eval_cache = (int)v;
    if (v == 0) eval_drop_spaces();
  } else if (n == "replica_warps") {
    if (v != 1 && v != 2 && v != 4 && v != 8) return fail(GD_E_INVALID, "replica_warps = %lld (1, 2, 4 or 8)", v);
    g_opt.replica_warps = (int)v;
  } else if (n == "dock_device_pack") {
    if (v != 0 && v != 1) return fail(GD_E_INVALID, "dock_device_pack = %lld", v);
    g_opt.dock_device_pack = (int)v;
  } else if (n == "dock_record_direct") {
    if (v != 0 && v != 1) return fail(GD_E_INVALID, "dock_record_direct = %lld", v);
    g_opt.dock_record_direct = (int)v;
  } else if (n == "device_base") {
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess) count = 0;
    if (v < 0 || (count > 0 && v >= count)) return fail(GD_E_INVALID, "device_base = %lld (%d devices)", v, count);
    g_opt.device_base = (int)v;
  } else if (n == "wait_limit") {
    if (v < 0 || v > 0xffffffffLL) return fail(GD_E_INVALID, "wait_limit = %lld", v);
    g_opt.wait_limit = v;
  } else if (n == "stall_test") {
    if (v < 0 || v > 2) return fail(GD_E_INVALID, "stall_test = %lld", v);
    g_opt.stall_test = (int)v;
  } else if (n == "fail_alloc") {
    if (v < 0 || v > 1000000) return fail(GD_E_INVALID, "fail_alloc = %lld", v);
    set_injected_alloc_failures((int)v);
  } else if (n == "graph") {
    if (v != 0 && v != 1) return fail(GD_E_INVALID, "graph = %lld", v);
    g_opt.graph = (int)v;
  } else {
    return fail(GD_E_INVALID, "unknown option '%s'", name);
  }
  return GD_OK;
}

long long gd_get_option(const char *name)
{
  if (!name) return GD_E_INVALID;
  std::lock_guard<std::mutex> lk(g_mu);
  const std::string n(name);
  if (n == "kernel") return g_opt.kernel;
  if (n == "precision") return g_opt.precision;
  if (n == "warps") return g_opt.warps;
  if (n == "kpl") return g_opt.kpl;
  if (n == "ab") return g_opt.ab;
  if (n == "graph") return g_opt.graph;
  if (n == "stage") return g_opt.stage;
  if (n == "replica_warps") return g_opt.replica_warps;
  if (n == "dock_device_pack") return g_opt.dock_device_pack;
  if (n == "dock_record_direct") return g_opt.dock_record_direct;
  if (n == "dock_cache") return g_opt.dock_cache;
  if (n == "eval_cache") return g_opt.eval_cache;
  if (n == "wait_limit") return g_opt.wait_limit;
  if (n == "device_base") return g_opt.device_base;
  if (n == "stall_test") return g_opt.stall_test;
  if (n == "fail_alloc") return injected_alloc_failures();
  return GD_E_INVALID;
}

// ---------------------------------------------------------------- Dock --
int SetDevice(void)
{
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count < 1) return fail(GD_E_NODEVICE, "no CUDA device");
  const int n = ngpu();
  if (dev_of(n - 1) >= count)
    return fail(GD_E_NODEVICE, "%d GPUs from device %d requested, %d present", n, dev_of(0), count);
  for (int g = 0; g < n; ++g) {
    GD_CUDA(cudaSetDevice(dev_of(g)));
    GD_CUDA(cudaDeviceSetCacheConfig(cudaFuncCachePreferShared));  // prepair.C:11-20
  }
  return GD_OK;
}

int DeviceAlloc(Complex **cd, Record **rd, gd_rng_t **rng)
{
  if (!cd || !rd || !rng) return fail(GD_E_INVALID, "null argument");
  const int n = ngpu();
  for (int g = 0; g < n; ++g) {
    GD_CUDA(cudaSetDevice(dev_of(g)));
    cd[g] = nullptr;
    rd[g] = nullptr;
    if (cudaMalloc((void **)&cd[g], sizeof(Complex)) != cudaSuccess)
      return fail(GD_E_NOMEM, "device Complex (%zu B) on GPU %d", sizeof(Complex), g);
    if (cudaMalloc((void **)&rd[g], sizeof(Record) * (size_t)GD_MAX_REP) != cudaSuccess)
      return fail(GD_E_NOMEM, "device Record[%d] on GPU %d", GD_MAX_REP, g);
    rng[g] = new gd_rng;
  }
  return GD_OK;
}

int DeviceFree(Complex **cd, Record **rd, gd_rng_t **rng)
{
  if (!cd || !rd || !rng) return fail(GD_E_INVALID, "null argument");
  const int n = ngpu();
  for (int g = 0; g < n; ++g) {
    GD_CUDA(cudaSetDevice(dev_of(g)));
    if (rng[g] && rng[g]->dock) destroy(rng[g]->dock);
    if (cd[g]) GD_CUDA(cudaFree(cd[g]));
    if (rd[g]) GD_CUDA(cudaFree(rd[g]));
    delete rng[g];
    cd[g] = nullptr;
    rd[g] = nullptr;
    rng[g] = nullptr;
  }
  return GD_OK;
}

// Replicas per GPU of the split of prepair.C:366-392 (maximising balance);
// with replica exchange on, cut at protein-conformation blocks so that exchange
// partners (same protein and ligand conformation) stay on one GPU.
static int split_per_gpu(const Complex *ch, int n, int *per_out)
{
  const int n_rep = ch->size.n_rep;
  if (n < 1) return fail(GD_E_INVALID, "ngpu = %d", n);
  if (n_rep < 1 || n_rep > GD_MAX_REP) return fail(GD_E_INVALID, "n_rep = %d", n_rep);
  int per = (n_rep + n - 1) / n;
  const McPara &mp = ch->mcpara;
  const bool exch = mp.steps_per_exchange > 0 && ch->size.n_tmp > 1;
  if (exch && n > 1) {
    const int block = ch->size.n_tmp * ch->size.n_lig;
    per = ((ch->size.n_prt + n - 1) / n) * block;
  }
  const int n_active = (n_rep + per - 1) / per;
  if (n_active < n) return fail(GD_E_INVALID, "%d replicas cannot keep %d GPUs busy", n_rep, n);
  *per_out = per;
  return GD_OK;
}

int SetParaT(Complex *ch, ParaT **pt)
{
  if (!ch || !pt) return fail(GD_E_INVALID, "null argument");
  const int n = ngpu();
  const int n_rep = ch->size.n_rep;
  int per = 0;
  GD_TRY(split_per_gpu(ch, n, &per));
  for (int g = 0; g < n; ++g) {
    pt[g]->rep_begin = per * g;
    pt[g]->rep_end = std::min(pt[g]->rep_begin + per, n_rep) - 1;
    pt[g]->n_rep = pt[g]->rep_end - pt[g]->rep_begin + 1;
    pt[g]->record_sz = (int)sizeof(Record) * pt[g]->n_rep;
  }
  return GD_OK;
}

int gd_replica_range(const Complex *ch, int ngpu, int g, int *rep_begin, int *rep_end)
{
  if (!ch || !rep_begin || !rep_end) return fail(GD_E_INVALID, "null argument");
  if (g < 0 || g >= ngpu) return fail(GD_E_INVALID, "GPU %d of %d", g, ngpu);
  int per = 0;
  GD_TRY(split_per_gpu(ch, ngpu, &per));
  *rep_begin = per * g;
  *rep_end = std::min(*rep_begin + per, ch->size.n_rep) - 1;
  return GD_OK;
}

int gd_ensemble_create_complex_range(const Complex *cx, int rep_begin, int rep_end, uint64_t seed, int device,
                                     gd_ensemble_t **out)
{
  if (!out || !cx) return fail(GD_E_INVALID, "null argument");
  *out = nullptr;
  if (rep_begin < 0 || rep_end < rep_begin || rep_end >= cx->size.n_rep)
    return fail(GD_E_INVALID, "replica range [%d, %d] of %d", rep_begin, rep_end, cx->size.n_rep);
  gd_ensemble *e = nullptr;
  GD_TRY(ensemble_from_complex_range(cx, rep_begin, rep_end, seed, nullptr, device, &e));
  *out = e;
  return GD_OK;
}

int CopyH2D(Complex *ch, Complex **cd, ParaT **pt)
{
  if (!ch || !cd || !pt) return fail(GD_E_INVALID, "null argument");
  const int n = ngpu();
  for (int g = 0; g < n; ++g) {
    GD_CUDA(cudaSetDevice(dev_of(g)));
    ch->rep_begin = pt[g]->rep_begin;  // prepair.C:119-123
    ch->rep_end = pt[g]->rep_end;
    GD_CUDA(cudaMemcpy(cd[g], ch, sizeof(Complex), cudaMemcpyHostToDevice));
  }
  return GD_OK;
}

int InitCurand(gd_rng_t **rng)
{
  if (!rng) return fail(GD_E_INVALID, "null argument");
  const int n = ngpu();
  const char *env = std::getenv("GDOCK_SEED");
  const uint64_t base = env ? std::strtoull(env, nullptr, 10) : (uint64_t)std::time(nullptr);
  for (int g = 0; g < n; ++g) {
    if (!rng[g]) return fail(GD_E_STATE, "InitCurand before DeviceAlloc");
    if (!rng[g]->seeded) {
      rng[g]->seed = base + (uint64_t)g;  // backend_gpu.cu:52-56: one seed per GPU
      rng[g]->seeded = 1;
    }
    rng[g]->calls = 0;
  }
  return GD_OK;
}

int gd_rng_dock_reuse(const gd_rng_t *rng, uint64_t *calls, uint64_t *reused)
{
  if (!rng || !calls || !reused) return fail(GD_E_INVALID, "null argument");
  *calls = rng->dock_calls;
  *reused = rng->dock_reused;
  return GD_OK;
}

int gd_rng_seed(gd_rng_t *rng, uint64_t seed)
{
  if (!rng) return fail(GD_E_INVALID, "null rng");
  rng->seed = seed;
  rng->seeded = 1;
  rng->calls = 0;
  return GD_OK;
}

int Dock(Complex *ch, Record *rh, Complex **cd, Record **rd, ParaT **pt, gd_rng_t **rng)
{
  if (!ch || !rh || !cd || !rd || !pt || !rng) return fail(GD_E_INVALID, "null argument");
  const int n = ngpu();
  const McPara &mp = ch->mcpara;
  const int steps_total = mp.steps_total, spd = mp.steps_per_dump;
  if (steps_total < 0) return fail(GD_E_INVALID, "steps_total = %d", steps_total);
  if (spd < 1 || spd > GD_STEPS_PER_DUMP)
    return fail(GD_E_INVALID, "steps_per_dump = %d outside [1, %d] (Record capacity)", spd, GD_STEPS_PER_DUMP);
  const int spx = (mp.steps_per_exchange > 0 && ch->size.n_tmp > 1) ? mp.steps_per_exchange : 0;
  std::vector<gd_ensemble *> ens(n, nullptr);
  // where the kernels write the Records: the device array rd[g], copied to rh after each
  // chunk (backend_gpu.cu:108-110), or, when rh is page-locked host memory this GPU can
  // address (cudaHostAlloc, or cudaHostRegister with mapping), rh itself: each entry then
  // crosses PCIe as the kernel writes it, while the chunk runs, and no copy follows
  std::vector<Record *> rdst(n, nullptr);
  std::vector<char> direct(n, 0);
  const bool try_direct = opts().dock_record_direct != 0;
  int rc = GD_OK;
  Tracer tr("Dock");
  for (int g = 0; g < n && rc == GD_OK; ++g) {
    if (!rng[g] || !cd[g] || !rd[g]) {
      rc = fail(GD_E_STATE, "Dock before DeviceAlloc/InitCurand on GPU %d", g);
      break;
    }
    rdst[g] = rd[g];
    if (try_direct && (rc = set_device(dev_of(g))) == GD_OK) {
      cudaPointerAttributes at{};
      if (cudaPointerGetAttributes(&at, rh + pt[g]->rep_begin) == cudaSuccess && at.type == cudaMemoryTypeHost &&
          at.devicePointer != nullptr) {
        rdst[g] = (Record *)at.devicePointer;
        direct[g] = 1;
      } else {
        (void)cudaGetLastError();  // pageable memory: the copy below
      }
    }
    if (rc != GD_OK) break;
    // each Dock call draws a fresh stream from the handle (the reference's curand state advances)
    const uint64_t seed = rng[g]->seed + (rng[g]->calls++ << 32);
    rc = dock_ensemble(rng[g], ch, cd[g], pt[g]->rep_begin, pt[g]->rep_end, seed, rdst[g], dev_of(g), &ens[g]);
  }
  tr.mark("pack+create");
  // initial energy, backend_gpu.cu:87-91: one step, no move, forced accept
  for (int g = 0; g < n && rc == GD_OK; ++g) {
    rc = set_device(dev_of(g));
    if (rc == GD_OK) rc = launch_mc(ens[g], 0, 1, kMcInitial | kMcRecord | kMcResetRecord | kMcStoreAccept);
  }
  tr.mark("initial (enqueued)");
  // dump chunks, backend_gpu.cu:96-114
  for (int s1 = 0; s1 < steps_total && rc == GD_OK; s1 += spd) {
    for (int g = 0; g < n && rc == GD_OK; ++g) {
      rc = set_device(dev_of(g));
      ens[g]->step = s1;
      if (rc == GD_OK) rc = advance(ens[g], spd, spx, kMcResetRecord, kMcRecord, kMcStoreAccept);
    }
    for (int g = 0; g < n && rc == GD_OK; ++g) {
      rc = set_device(dev_of(g));
      if (rc != GD_OK) break;
      const cudaError_t ce =
          direct[g] ? cudaSuccess
                    : cudaMemcpyAsync(rh + pt[g]->rep_begin, rd[g], sizeof(Record) * (size_t)pt[g]->n_rep,
                                      cudaMemcpyDeviceToHost, ens[g]->st);
      if (ce == cudaSuccess) {
        const cudaError_t se = cudaStreamSynchronize(ens[g]->st);
        if (se != cudaSuccess) rc = fail(GD_E_CUDA, "Dock: %s", cudaGetErrorString(se));
      } else {
        rc = fail(GD_E_CUDA, "Dock record copy: %s", cudaGetErrorString(ce));
      }
      if (rc == GD_OK) rc = check_err(ens[g]);
    }
    tr.mark("chunk + record copy");
  }
  // final replica states: device Complex (as the reference) and the host Complex
  for (int g = 0; g < n && rc == GD_OK; ++g) {
    rc = set_device(dev_of(g));
    if (rc != GD_OK) break;
    const DevJob &J = ens[g]->jobs[0].dj;
    const size_t bytes = sizeof(ReplicaMC) * (size_t)J.nrep;
    if (cudaMemcpyAsync(cd[g]->replica + pt[g]->rep_begin, J.rep, bytes, cudaMemcpyDeviceToDevice, ens[g]->st) !=
            cudaSuccess ||
        cudaMemcpyAsync(ch->replica + pt[g]->rep_begin, J.rep, bytes, cudaMemcpyDeviceToHost, ens[g]->st) !=
            cudaSuccess ||
        cudaStreamSynchronize(ens[g]->st) != cudaSuccess)
      rc = fail(GD_E_CUDA, "Dock final copy on GPU %d", g);
  }
  tr.mark("final replica copy");
  for (int g = 0; g < n; ++g)
    if (ens[g] && (!rng[g] || rng[g]->dock != ens[g])) destroy(ens[g]);  // not cached
  if (rc != GD_OK)
    for (int g = 0; g < n; ++g)
      if (rng[g] && rng[g]->dock) {  // drop the cached state of a failed call
        destroy(rng[g]->dock);
        rng[g]->dock = nullptr;
        rng[g]->dock_prt.clear();
      }
  return rc;
}

}  // extern "C"

// ------------------------------------------------------------ poses --
namespace {

// Launch shape of n poses: a team of warps per pose where one wave holds them
// (gd_shape.cu); else one warp each, spread over the SMs where one wave holds
// that; else with the pocket staged in shared memory or read through L1 and the
// poses per CTA that keep the most poses in flight (ties: staged, 8 poses).  A
// 64-atom ligand against 3000 points staged is 136 KB a CTA, so one CTA of 8 warps
// per SM: 16384 poses 6.26 ms; through L1 three CTAs fit, 24 warps: 3.96 ms (FP64,
// 2048 poses on 8 and 16 warps: 8.89 and 5.12 ms).
int eval_shape(const ShapeQuery &q, int n, TileConfig &tc, int &grid)
{
  // (one wave holds at most 12 teams of two and 24 warps per SM)
  if ((n <= 16 * q.nsm && choose_team(q, tc, grid)) || (n <= 32 * q.nsm && choose_spread(q, tc, grid))) return GD_OK;
  long long flight = 0;
  int occ = 0;
  for (const int staged : {1, 0})
    for (int w : {8, 12, 16, 4, 2, 1}) {
      if (staged && q.stage_opt == 0) continue;
      TileConfig t = tc;
      t.warps_per_cta = w;
      t.stage = staged;
      const size_t ts = q.smem(t);
      if (ts > kSmemLimit) continue;
      const int to = kernel_occupancy(q.mode, q.precision, t, ts);
      const long long fl = std::min<long long>(n, (long long)to * w * q.nsm);
      if (fl <= flight) continue;
      flight = fl;
      tc = t;
      occ = to;
    }
  if (occ < 1) return fail(GD_E_CAPACITY, "ligand slots too large for shared memory");
  grid = occ * q.nsm;
  return GD_OK;
}

// The poses of a call in the order they run, grouped by protein conformation so
// that a CTA meets one; empty: as they are.
std::vector<int> eval_order(int n, const int *conf, int nprt)
{
  std::vector<int> at(nprt + 1, 0), ord;
  bool sorted = true;
  for (size_t i = 0; i < (size_t)n; ++i) {
    ++at[conf[2 * i + 1] + 1];
    sorted &= i == 0 || conf[2 * i + 1] >= conf[2 * i - 1];
  }
  if (sorted) return ord;
  for (int p = 0; p < nprt; ++p) at[p + 1] += at[p];
  ord.resize(n);
  for (int i = 0; i < n; ++i) ord[at[conf[2 * (size_t)i + 1]]++] = i;
  return ord;
}

// What a call sends (conformations, poses, work items) and gets back (energies,
// raw terms, energies in FP64, the error words), each side in one piece: its
// places in the device block and in the host copy of it.
struct EvalBlock {
  size_t conf, mm, items, sent, out, raw, out64, err, end;
  int n;
  EvalBlock(int n_, size_t nitem, bool with_raw, bool with_64) : n(n_)
  {
    size_t off = 0;
    auto take = [&off](size_t bytes) {
      const size_t o = off;
      off = (off + bytes + 255) & ~(size_t)255;
      return o;
    };
    conf = take(sizeof(int) * 2 * n);
    mm = take(sizeof(float) * 6 * n);
    items = take(sizeof(WorkItem) * nitem);
    sent = off;
    out = take(sizeof(float) * 10 * n);
    raw = take(with_raw ? sizeof(float) * 9 * n : 0);
    out64 = take(with_64 ? sizeof(double) * 10 * n : 0);
    err = take(4 * sizeof(int));
    end = off;
  }
  void send(unsigned char *h, const std::vector<int> &ord, const int *c, const float *m) const
  {
    if (ord.empty()) {
      std::memcpy(h + conf, c, sizeof(int) * 2 * n);
      std::memcpy(h + mm, m, sizeof(float) * 6 * n);
      return;
    }
    int *hc = (int *)(h + conf);
    float *hm = (float *)(h + mm);
    for (int i = 0; i < n; ++i) {
      std::memcpy(hc + 2 * (size_t)i, c + 2 * (size_t)ord[i], sizeof(int) * 2);
      std::memcpy(hm + 6 * (size_t)i, m + 6 * (size_t)ord[i], sizeof(float) * 6);
    }
  }
  template <typename T>
  void back(const unsigned char *h, size_t at, const std::vector<int> &ord, T *to, int k) const
  {
    const T *from = (const T *)(h + at);
    if (ord.empty()) {
      std::memcpy(to, from, sizeof(T) * k * n);
      return;
    }
    for (int i = 0; i < n; ++i) std::memcpy(to + (size_t)k * ord[i], from + (size_t)k * i, sizeof(T) * k);
  }
  void bind(KArgs &a, unsigned char *d, bool with_raw, bool with_64) const
  {
    a.conf = (const int *)(d + conf);
    a.mm = (const float *)(d + mm);
    a.out = (float *)(d + out);
    a.raw = with_raw ? (float *)(d + raw) : nullptr;
    a.out64 = with_64 ? (double *)(d + out64) : nullptr;
  }
};

// Energies of n poses of job `job` of a resident ensemble (mode 1 of the batched kernel).  The device and host blocks
// of a call stay with the ensemble up to kEvalKeep bytes each: one copy each way and no allocation in the calls after.
int eval_on(gd_ensemble *e, int job, int n, const int *conf, const float *mm, int precision, float *out,
            double *out64, float *raw)
{
  const DevJob &J = e->jobs[job].dj;
  for (size_t i = 0; i < (size_t)n; ++i)
    if (conf[2 * i] < 0 || conf[2 * i] >= J.nlig || conf[2 * i + 1] < 0 || conf[2 * i + 1] >= J.nprt)
      return fail(GD_E_INVALID, "pose %zu: conformation (%d, %d) out of range", i, conf[2 * i], conf[2 * i + 1]);
  const Options o = opts();
  TileConfig tc{8, o.kpl, o.ab};
  default_pair_tile(tc.kpl, tc.ab);
  if (precision == GD_PREC_FP64) tc.kpl = 1, tc.ab = 8;
  const std::vector<int> ord = eval_order(n, conf, J.nprt);
  std::vector<int> count(J.nprt, 0);
  for (size_t i = 0; i < (size_t)n; ++i) ++count[conf[2 * i + 1]];
  ShapeQuery q;
  GD_CUDA(cudaDeviceGetAttribute(&q.nsm, cudaDevAttrMultiProcessorCount, e->device));
  q.mode = 1;
  q.precision = precision;
  q.Pmax = e->Pmax;
  q.lig_slots = e->lig_slots;
  q.items = [&](int R) {
    long long m = 0;
    for (const long long k : count) m += (k + R - 1) / R;
    return m;
  };
  int grid = 0;
  GD_TRY(eval_shape(q, n, tc, grid));
  const int R = tc.warps_per_cta / tc.group;  // poses per CTA
  const size_t nitem = (size_t)q.items(R);
  const EvalBlock B(n, nitem, raw != nullptr, out64 != nullptr);
  if (B.end > e->eval_bytes) {
    cudaFree(e->eval_dev);
    e->eval_dev = nullptr;
    e->eval_bytes = 0;
    GD_CUDA(cudaMalloc(&e->eval_dev, B.end));
    e->eval_host.reset(new unsigned char[B.end]);
    e->eval_bytes = B.end;
  }
  unsigned char *h = e->eval_host.get(), *d = e->eval_dev;
  B.send(h, ord, conf, mm);
  WorkItem *it = (WorkItem *)(h + B.items);
  for (int p = 0, r = 0; p < J.nprt; r += count[p++])
    for (long long k = 0; k < count[p]; k += R) *it++ = WorkItem{job, p, (int)(r + k), (int)std::min<long long>(R, count[p] - k)};
  GD_CUDA(cudaMemcpyAsync(d, h, B.sent, cudaMemcpyHostToDevice, e->st));
  GD_CUDA(cudaMemsetAsync(e->d_queue, 0, sizeof(int), e->st));
  KArgs a{};
  a.jobs = e->d_jobs;
  a.items = (const WorkItem *)(d + B.items);
  a.n_items = (int)nitem;
  a.queue = e->d_queue;
  a.err = e->d_err;
  a.P = tc.stage ? e->Pmax : 0;
  a.Pall = e->Pmax;
  a.lig_slots = e->lig_slots;
  B.bind(a, d, raw != nullptr, out64 != nullptr);
  GD_CUDA(launch_kernel(1, precision, tc, a, std::max(1, std::min((int)nitem, grid)), e->st));
  GD_CUDA(cudaMemcpyAsync(h + B.out, d + B.out, B.err - B.out, cudaMemcpyDeviceToHost, e->st));
  GD_CUDA(cudaStreamSynchronize(e->st));
  B.back(h, B.out, ord, out, 10);
  if (raw) B.back(h, B.raw, ord, raw, 9);
  if (out64) B.back(h, B.out64, ord, out64, 10);
  if (e->eval_bytes > kEvalKeep) {
    cudaFree(e->eval_dev);
    e->eval_dev = nullptr;
    e->eval_host.reset();
    e->eval_bytes = 0;
  }
  return check_err(e);
}

// The driver's calls about contexts, looked up in it; ok: all are there.
struct ContextCalls {
  CUresult (*get)(CUcontext *) = nullptr;
  CUresult (*set)(CUcontext) = nullptr;
  CUresult (*state)(CUdevice, unsigned *, int *) = nullptr;
  CUresult (*retain)(CUcontext *, CUdevice) = nullptr;
  CUresult (*release)(CUdevice) = nullptr;
  CUresult (*id)(CUcontext, unsigned long long *) = nullptr;
  bool ok = false;
  ContextCalls()
  {
    auto find = [](const char *name, auto &f) {
      void *p = nullptr;
      cudaDriverEntryPointQueryResult q;
      if (cudaGetDriverEntryPointByVersion(name, &p, 12000, cudaEnableDefault, &q) != cudaSuccess) p = nullptr;
      f = reinterpret_cast<std::remove_reference_t<decltype(f)>>(p);
      return p != nullptr;
    };
    ok = find("cuCtxGetCurrent", get) && find("cuCtxSetCurrent", set) && find("cuDevicePrimaryCtxGetState", state) &&
         find("cuDevicePrimaryCtxRetain", retain) && find("cuDevicePrimaryCtxRelease", release) && find("cuCtxGetId", id);
  }
  static const ContextCalls &get_calls()
  {
    static const ContextCalls c;
    return c;
  }
};

// The id of device dev's primary context (no two contexts of a process have the same; a reset context's successor has
// another), 0 where there is none or the driver does not tell.  With `current`, 0 too where the calling thread's context
// is another one (a thread without one gets the primary one from the runtime).
unsigned long long primary_context(int dev, bool current)
{
  const ContextCalls &d = ContextCalls::get_calls();
  unsigned flags = 0;
  int active = 0;
  CUcontext c = nullptr, p = nullptr;
  unsigned long long id = 0;
  if (!d.ok || d.state(dev, &flags, &active) != CUDA_SUCCESS || !active) return 0;
  if (current && d.get(&c) != CUDA_SUCCESS) return 0;
  if (d.retain(&p, dev) != CUDA_SUCCESS) return 0;
  if ((c && c != p) || d.id(p, &id) != CUDA_SUCCESS) id = 0;
  d.release(dev);
  return id;
}

// A device block and a stream for one call, from those that calls before it left (option "eval_cache"): getting and
// giving back 10 MB and a stream takes 750 us, four times what a call of 64 poses does with them.  At most
// kEvalSpaces are kept, of kEvalKeep bytes each at most; a call that needs more, or fails, leaves none, nor
// does one in another context than the device's primary one.  A block of a context that has been reset is forgotten.
struct EvalSpace {
  struct Kept {
    int dev;
    unsigned long long ctx;
    size_t bytes;
    unsigned char *d;
    cudaStream_t st;
  };
  static constexpr size_t kEvalSpaces = 4;
  static std::mutex mu;
  static std::vector<Kept> kept;

  int dev;
  unsigned long long ctx;  // 0: not one whose blocks are kept
  size_t bytes;
  unsigned char *d = nullptr;
  cudaStream_t st = nullptr;
  bool good = false;  // set by the call when all its work on the stream is done and was right

  EvalSpace(int dev_, size_t need) : dev(dev_), ctx(0), bytes(need)
  {
    ctx = primary_context(dev, true);
    if (ctx) {
      std::lock_guard<std::mutex> lk(mu);
      kept.erase(std::remove_if(kept.begin(), kept.end(), [this](const Kept &k) { return k.dev == dev && k.ctx != ctx; }),
                 kept.end());
      for (size_t i = 0; i < kept.size() && !d; ++i)
        if (kept[i].dev == dev && kept[i].bytes >= need) {
          bytes = kept[i].bytes;
          d = kept[i].d;
          st = kept[i].st;
          kept.erase(kept.begin() + i);
        }
    }
    if (d) return;
    if (cudaMalloc(&d, bytes) != cudaSuccess) d = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) st = nullptr;
    if (!ctx) ctx = primary_context(dev, true);  // the process's first call: the allocation has made the context
  }
  ~EvalSpace()
  {
    if (good && ctx && bytes <= kEvalKeep && opts().eval_cache) {
      std::lock_guard<std::mutex> lk(mu);
      // the smallest goes first, so that the sizes in use are the ones kept
      if (kept.size() == kEvalSpaces) {
        size_t k = 0;
        for (size_t i = 1; i < kept.size(); ++i)
          if (kept[i].bytes < kept[k].bytes) k = i;
        if (kept[k].bytes < bytes) {
          drop_kept(kept[k]);
          kept.erase(kept.begin() + k);
        }
      }
      if (kept.size() < kEvalSpaces) {
        kept.push_back(Kept{dev, ctx, bytes, d, st});
        return;
      }
    }
    drop(d, st);
    (void)cudaGetLastError();  // a failure here is the general path's to report
  }
  static void drop(unsigned char *d, cudaStream_t st)
  {
    if (st) cudaStreamSynchronize(st), cudaStreamDestroy(st);
    if (d) cudaFree(d);
  }
  static void drop_kept(const Kept &k)
  {
    if (primary_context(k.dev, false) != k.ctx) return;
    CUcontext c = nullptr;
    const ContextCalls &d = ContextCalls::get_calls();
    if (d.get(&c) == CUDA_SUCCESS && cudaSetDevice(k.dev) == cudaSuccess) drop(k.d, k.st);
    d.set(c);
  }
  static void drop_all()
  {
    std::lock_guard<std::mutex> lk(mu);
    for (const Kept &k : kept) drop_kept(k);
    kept.clear();
    (void)cudaGetLastError();
  }
};
std::mutex EvalSpace::mu;
std::vector<EvalSpace::Kept> EvalSpace::kept;

// Poses of a Complex in host memory, packed on the GPU (gd_devpack.cu) from the parts of it that the packing reads, in
// one allocation, and run as mode 2.  Returns false where eval_complex_host below is the one to answer: a size or a
// value that is not valid (its messages), another pair tile or test hook asked for, a CUDA error.
//
// 64 poses of 40 atoms x 1500 points x 11 conformations: 2.96 ms with the host packer, 0.19 ms here (sending 1.2 MB of
// the Complex 95 us, the two kernels 65).
bool eval_complex(const Complex *c, int n, const int *conf, const float *mm, int precision, float *out, double *out64,
                  float *raw)
{
  const ComplexSize &sz = c->size;
  auto in = [](int v, int lo, int hi) { return v >= lo && v <= hi; };
  const int L = c->lig[0].lig_natom, K = sz.kde_npoint, M = sz.mcs_nrow;
  if (!in(sz.n_lig, 1, GD_MAX_CONF_LIG) || !in(sz.n_prt, 1, GD_MAX_CONF_PRT) || !in(sz.n_tmp, 1, GD_MAX_TMP) ||
      !in(sz.n_rep, 1, GD_MAX_REP) || !in(L, 1, GD_MAXLIG) || !in(K, 0, GD_MAXKDE) || !in(M, 1, GD_MAX_MCS_ROW))
    return false;
  for (int i = 0; i < sz.n_lig; ++i)
    if (c->lig[i].lig_natom != L) return false;
  int P = 0;
  for (int i = 0; i < sz.n_prt; ++i) {
    if (!in(c->prt[i].prt_npoint, 1, GD_MAXPRO)) return false;
    P = std::max(P, c->prt[i].prt_npoint);
  }
  P = (P + kPointAlign - 1) / kPointAlign * kPointAlign;
  const ReplicaMC &r0 = c->replica[0];  // the general path reads the first replica
  if (!in(r0.idx_lig, 0, sz.n_lig - 1) || !in(r0.idx_prt, 0, sz.n_prt - 1) || !in(r0.idx_tmp, 0, sz.n_tmp - 1))
    return false;
  const Options o = opts();
  TileConfig tc{8, o.kpl, o.ab};
  default_pair_tile(tc.kpl, tc.ab);
  if (precision == GD_PREC_FP64) tc.kpl = 1, tc.ab = 8;
  else if (tc.kpl != 4 || tc.ab != 8) return false;
  if (injected_alloc_failures() > 0) return false;

  int dev = 0;
  ShapeQuery q;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&q.nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return false;
  q.mode = 2;
  q.precision = precision;
  q.Pmax = P;
  q.lig_slots = (L + 3) & ~3;
  q.stage_opt = 0;
  q.items = [n](int R) { return ((long long)n + R - 1) / R; };
  int grid = 0;
  if (eval_shape(q, n, tc, grid) != GD_OK) return false;
  const int R = tc.warps_per_cta / tc.group;
  const std::vector<int> ord = eval_order(n, conf, sz.n_prt);
  const EvalBlock B(n, 0, raw != nullptr, out64 != nullptr);

  // the block: the call's data, the Complex, the packed job
  size_t off = B.end;
  auto take = [&off](size_t bytes) {
    const size_t p = off;
    off = (off + bytes + 255) & ~(size_t)255;
    return p;
  };
  const size_t at_cx = take(offsetof(Complex, lig_file)), at_job = take(sizeof(DevJob)), at_par = take(sizeof(DevParams)),
               at_ref = take(sizeof(float4) * kLigTypes * kTabCols), at_lgrp = take(sizeof(int2) * GD_MAXLIG),
               at_lcen = take(sizeof(float) * 3 * sz.n_lig), at_pcen = take(sizeof(float) * 3 * sz.n_prt),
               at_tcc = take(sizeof(float) * M), at_lig = take(sizeof(float4) * ((L + 3) & ~3) * sz.n_lig),
               at_kde = take(sizeof(int4) * 2 * std::max(K, 1)), at_mcs = take(sizeof(float4) * L * M),
               at_pos = take(sizeof(float4) * P * sz.n_prt), at_aux = take(sizeof(float2) * P * sz.n_prt),
               at_ncdc = take(sizeof(int) * sz.n_prt), at_cnt = take(sizeof(int) * sz.n_prt);
  const int stride = std::min(kLigTypes, L) * P;
  const size_t at_cell = take(sizeof(int) * (size_t)stride * sz.n_prt);

  EvalSpace H(dev, off);
  if (!H.d || !H.st) return false;
  std::unique_ptr<unsigned char[]> host(new unsigned char[B.end]);
  unsigned char *h = host.get(), *d = H.d;
  B.send(h, ord, conf, mm);
  std::memset(h + B.err, 0, 4 * sizeof(int));
  auto up = [&](const void *from, size_t bytes) {
    const size_t at = (const unsigned char *)from - (const unsigned char *)c;
    return cudaMemcpyAsync(d + at_cx + at, from, bytes, cudaMemcpyHostToDevice, H.st) == cudaSuccess;
  };
  const size_t kde_row = sizeof(c->kde.t), at_kt = (const unsigned char *)c->kde.t - (const unsigned char *)c;
  bool ok = cudaMemcpyAsync(d, h, B.sent, cudaMemcpyHostToDevice, H.st) == cudaSuccess &&
            cudaMemcpyAsync(d + B.err, h + B.err, 4 * sizeof(int), cudaMemcpyHostToDevice, H.st) == cudaSuccess &&
            up(c->lig, sizeof(c->lig[0]) * sz.n_lig) && up(c->prt, sizeof(c->prt[0]) * sz.n_prt) &&
            up(c->psp.psp, sizeof(c->psp.psp[0]) * kLigTypes) && up(c->mcs, sizeof(c->mcs[0]) * M) &&
            up(&c->enepara, sizeof(c->enepara)) && up(&c->size, offsetof(Complex, lig_file) - offsetof(Complex, size)) &&
            (K == 0 || cudaMemcpy2DAsync(d + at_cx + at_kt, kde_row, c->kde.t, kde_row, sizeof(float) * K, 4,
                                         cudaMemcpyHostToDevice, H.st) == cudaSuccess);
  PackDst D{};
  D.job = (DevJob *)(d + at_job);
  D.par = (DevParams *)(d + at_par);
  D.ref4 = (float4 *)(d + at_ref);
  D.err = (int *)(d + B.err);
  D.lgrp = (int2 *)(d + at_lgrp);
  D.lcenter = (float *)(d + at_lcen);
  D.pcenter = (float *)(d + at_pcen);
  D.tcc = (float *)(d + at_tcc);
  D.lig = (float4 *)(d + at_lig);
  D.kslot = (int4 *)(d + at_kde);
  D.mcs = (float4 *)(d + at_mcs);
  D.pos = (float4 *)(d + at_pos);
  D.aux = (float2 *)(d + at_aux);
  D.ncdc = (int *)(d + at_ncdc);
  D.pcell_cnt = (int *)(d + at_cnt);
  D.pcell4 = (int *)(d + at_cell);
  D.pcell_stride = stride;
  D.kde_cap = std::max(K, 1);
  D.Ppad = P;
  D.nkde_expect = -1;
  D.expect_L = L;
  D.expect_nlig = sz.n_lig;
  D.expect_nprt = sz.n_prt;
  D.expect_M = M;
  D.expect_ntmp = -1;
  ok = ok && device_pack((const Complex *)(d + at_cx), D, H.st) == cudaSuccess;
  KArgs a{};
  a.jobs = D.job;
  a.err = D.err;
  a.Pall = P;
  a.lig_slots = q.lig_slots;
  a.n_poses = n;
  a.n_items = (int)q.items(R);
  B.bind(a, d, raw != nullptr, out64 != nullptr);
  ok = ok && launch_kernel(2, precision, tc, a, std::min(a.n_items, grid), H.st) == cudaSuccess &&
       cudaMemcpyAsync(h + B.out, d + B.out, B.end - B.out, cudaMemcpyDeviceToHost, H.st) == cudaSuccess &&
       cudaStreamSynchronize(H.st) == cudaSuccess;
  int err = 0;
  std::memcpy(&err, h + B.err, sizeof(err));
  H.good = ok;
  if (!ok || err != 0) return false;
  B.back(h, B.out, ord, out, 10);
  if (raw) B.back(h, B.raw, ord, raw, 9);
  if (out64) B.back(h, B.out64, ord, out64, 10);
  return true;
}

// The same with the host packer, as an ensemble of one job.
int eval_complex_host(const Complex *c, int n, const int *conf, const float *mm, int precision, float *out,
                      double *out64, float *raw, int dev)
{
  PocketData pk;
  JobData jd;
  GD_TRY(pocket_from_complex(c, pk));
  GD_TRY(job_from_complex(c, 0, 0, 0, jd));
  gd_ensemble *e = new gd_ensemble;
  e->device = dev;
  e->pockets.resize(1);
  e->jobs.resize(1);
  int rc = pack_pocket(pk, e->pockets[0]);
  if (rc == GD_OK) rc = pack_job(jd, e->pockets[0], c->enepara, false, nullptr, e->jobs[0]);
  if (rc == GD_OK) {
    const DevJob &J = e->jobs[0].dj;
    e->precision = precision;
    e->Pmax = J.npoint_pad;
    e->lig_slots = (J.natom + 3) & ~3;
    rc = upload_jobs(e);
  }
  if (rc == GD_OK && cudaMalloc(&e->d_queue, sizeof(int)) != cudaSuccess) rc = fail(GD_E_CUDA, "cudaMalloc");
  // error words as an ensemble's: kernel flags, then the device packer's details
  if (rc == GD_OK && cudaMalloc(&e->d_err, 4 * sizeof(int)) != cudaSuccess) rc = fail(GD_E_CUDA, "cudaMalloc");
  if (rc == GD_OK && cudaMemset(e->d_err, 0, 4 * sizeof(int)) != cudaSuccess) rc = fail(GD_E_CUDA, "cudaMemset");
  if (rc == GD_OK && cudaStreamCreateWithFlags(&e->st, cudaStreamNonBlocking) != cudaSuccess)
    rc = fail(GD_E_CUDA, "cudaStreamCreate");
  if (rc == GD_OK) rc = eval_on(e, 0, n, conf, mm, precision, out, out64, raw);
  destroy(e);
  return rc;
}

}  // namespace

void eval_drop_spaces() { EvalSpace::drop_all(); }

extern "C" {

int gd_eval_poses(const Complex *c, int n, const int *conf, const float *mm, int precision, float *out,
                  double *out64, float *raw)
{
  if (!c || n < 0 || (n > 0 && (!conf || !mm || !out))) return fail(GD_E_INVALID, "null argument");
  if (precision < GD_PREC_FP32 || precision > GD_PREC_FP64) return fail(GD_E_INVALID, "precision = %d", precision);
  if (n == 0) return GD_OK;
  for (size_t i = 0; i < (size_t)n; ++i)
    if (conf[2 * i] < 0 || conf[2 * i] >= c->size.n_lig || conf[2 * i + 1] < 0 || conf[2 * i + 1] >= c->size.n_prt)
      return fail(GD_E_INVALID, "pose %zu: conformation (%d, %d) out of range", i, conf[2 * i], conf[2 * i + 1]);
  int dev = 0;
  GD_CUDA(cudaGetDevice(&dev));
  if (eval_complex(c, n, conf, mm, precision, out, out64, raw)) return GD_OK;
  return eval_complex_host(c, n, conf, mm, precision, out, out64, raw, dev);
}

// ---------------------------------------------------------- ensembles --
int gd_ensemble_create(const gd_pocket_desc_t *pockets, int npocket, const gd_job_desc_t *jobs, int njob,
                       const EnePara *enepara, int device, gd_ensemble_t **out)
{
  if (!out) return fail(GD_E_INVALID, "null out");
  *out = nullptr;
  if (!pockets || npocket < 1 || !jobs || njob < 1 || !enepara) return fail(GD_E_INVALID, "empty ensemble");
  GD_TRY(set_device(device));
  gd_ensemble *e = new gd_ensemble;
  e->device = device;
  e->pockets.resize(npocket);
  e->jobs.resize(njob);
  e->rep_prt.resize(njob);
  int rc = GD_OK;
  std::vector<int> nconf(npocket);
  for (int p = 0; p < npocket && rc == GD_OK; ++p) {
    PocketData pk;
    rc = pocket_from_desc(pockets[p], pk);
    pk.hdb_types = hdb_point_types(*enepara);
    if (rc == GD_OK) rc = pack_pocket(pk, e->pockets[p]);
    nconf[p] = pockets[p].nconf;
  }
  for (int j = 0; j < njob && rc == GD_OK; ++j) {
    const int p = jobs[j].pocket;
    if (p < 0 || p >= npocket) {
      rc = fail(GD_E_INVALID, "job %d: pocket %d out of range", j, p);
      break;
    }
    JobData jd;
    rc = job_from_desc(jobs[j], nconf[p], jd);
    if (rc == GD_OK) rc = pack_job(jd, e->pockets[p], *enepara, false, nullptr, e->jobs[j]);
    if (rc == GD_OK) read_replica_prt(e, j, jd.reps);
    e->jobs[j].pocket = p;
  }
  if (rc == GD_OK) rc = finish_create(e);
  if (rc != GD_OK) {
    destroy(e);
    return rc;
  }
  *out = e;
  return GD_OK;
}

int gd_ensemble_create_complex(const Complex *const *cx, int n, const uint64_t *seeds, int device,
                               gd_ensemble_t **out)
{
  if (!out) return fail(GD_E_INVALID, "null out");
  *out = nullptr;
  if (!cx || n < 1) return fail(GD_E_INVALID, "empty ensemble");
  GD_TRY(set_device(device));
  gd_ensemble *e = new gd_ensemble;
  e->device = device;
  e->jobs.resize(n);
  e->rep_prt.resize(n);
  std::vector<PocketData> seen;
  int rc = GD_OK;
  for (int j = 0; j < n && rc == GD_OK; ++j) {
    PocketData pk;
    JobData jd;
    rc = pocket_from_complex(cx[j], pk);
    if (rc == GD_OK) rc = job_from_complex(cx[j], 0, cx[j]->size.n_rep - 1, seeds ? seeds[j] : 0, jd);
    if (rc != GD_OK) break;
    // identical protein conformation sets share one device pocket
    int p = -1;
    for (size_t q = 0; q < seen.size(); ++q)
      if (seen[q].nconf == pk.nconf && seen[q].npts == pk.npts && seen[q].xyz == pk.xyz && seen[q].type == pk.type &&
          seen[q].cls == pk.cls && seen[q].cdc == pk.cdc && seen[q].seq3r == pk.seq3r && seen[q].hpp == pk.hpp &&
          seen[q].ele == pk.ele && seen[q].center == pk.center && seen[q].hdb_types == pk.hdb_types) {
        p = (int)q;
        break;
      }
    if (p < 0) {
      e->pockets.emplace_back();
      rc = pack_pocket(pk, e->pockets.back());
      seen.push_back(std::move(pk));
      p = (int)seen.size() - 1;
    }
    if (rc == GD_OK) rc = pack_job(jd, e->pockets[p], cx[j]->enepara, false, nullptr, e->jobs[j]);
    if (rc == GD_OK) read_replica_prt(e, j, jd.reps);
    e->jobs[j].pocket = p;
  }
  if (rc == GD_OK) rc = finish_create(e);
  if (rc != GD_OK) {
    destroy(e);
    return rc;
  }
  *out = e;
  return GD_OK;
}

int gd_ensemble_init(gd_ensemble_t *e)
{
  if (!e) return fail(GD_E_INVALID, "null ensemble");
  GD_TRY(set_device(e->device));
  return launch_mc(e, 0, 1, kMcInitial | kMcStoreAccept);
}

int gd_ensemble_run(gd_ensemble_t *e, int nsteps, int steps_per_exchange)
{
  if (!e) return fail(GD_E_INVALID, "null ensemble");
  if (nsteps < 0 || steps_per_exchange < 0) return fail(GD_E_INVALID, "nsteps = %d, steps_per_exchange = %d", nsteps, steps_per_exchange);
  GD_TRY(set_device(e->device));
  return advance(e, nsteps, steps_per_exchange, 0, 0, kMcStoreAccept);
}

int gd_ensemble_sync(gd_ensemble_t *e, double *kernel_ms, int *launches, int *all_launches)
{
  if (!e) return fail(GD_E_INVALID, "null ensemble");
  GD_TRY(set_device(e->device));
  GD_CUDA(cudaStreamSynchronize(e->st));
  double ms = 0;
  for (int i = 0; i + 1 < e->ev_used; i += 2) {
    float t = 0;
    GD_CUDA(cudaEventElapsedTime(&t, e->ev[i], e->ev[i + 1]));
    ms += t;
  }
  if (kernel_ms) *kernel_ms = ms;
  if (launches) *launches = e->launches;
  if (all_launches) *all_launches = e->all_launches;
  e->ev_used = 0;
  e->launches = 0;
  e->all_launches = 0;
  return check_err(e);
}

int gd_ensemble_num_replicas(const gd_ensemble_t *e, int job)
{
  if (!e || job < 0 || job >= (int)e->jobs.size()) return fail(GD_E_INVALID, "job %d", job);
  return e->jobs[job].dj.nrep;
}

int gd_ensemble_replicas(gd_ensemble_t *e, int job, ReplicaMC *out)
{
  if (!e || !out || job < 0 || job >= (int)e->jobs.size()) return fail(GD_E_INVALID, "job %d", job);
  GD_TRY(set_device(e->device));
  const DevJob &J = e->jobs[job].dj;
  GD_CUDA(cudaMemcpyAsync(out, J.rep, sizeof(ReplicaMC) * (size_t)J.nrep, cudaMemcpyDeviceToHost, e->st));
  GD_CUDA(cudaStreamSynchronize(e->st));
  return GD_OK;
}

int gd_ensemble_best_poses(gd_ensemble_t *e, int job, float *best_mm, double *best_energy)
{
  if (!e || job < 0 || job >= (int)e->jobs.size()) return fail(GD_E_INVALID, "job %d", job);
  GD_TRY(set_device(e->device));
  const DevJob &J = e->jobs[job].dj;
  std::vector<RepStats> s(J.nrep);
  GD_CUDA(cudaMemcpyAsync(s.data(), J.stats, sizeof(RepStats) * s.size(), cudaMemcpyDeviceToHost, e->st));
  GD_CUDA(cudaStreamSynchronize(e->st));
  for (int r = 0; r < J.nrep; ++r) {
    if (best_mm)
      for (int k = 0; k < 6; ++k) best_mm[6 * (size_t)r + k] = s[r].best_mm[k];
    if (best_energy) best_energy[r] = s[r].best_e;
  }
  return GD_OK;
}

int gd_ensemble_cluster(gd_ensemble_t *e, int job, int ref_lig, const float *ref_mm, float rmsd_cut,
                        gd_cluster_t *clusters, int max_clusters, int *n_clusters, int *cluster_of,
                        float *rmsd_to_ref)
{
  if (!e || job < 0 || job >= (int)e->jobs.size()) return fail(GD_E_INVALID, "job %d", job);
  if (!n_clusters || (max_clusters > 0 && !clusters) || max_clusters < 0) return fail(GD_E_INVALID, "null argument");
  GD_TRY(set_device(e->device));
  GD_CUDA(cudaStreamSynchronize(e->st));
  return cluster_job(e->jobs[job].dj, e->d_jobs + job, e->st, ref_lig, ref_mm, rmsd_cut, clusters, max_clusters,
                     n_clusters, cluster_of, rmsd_to_ref);
}

int gd_ensemble_eval_poses(gd_ensemble_t *e, int job, int n, const int *conf, const float *mm, int precision,
                           float *out, double *out64, float *raw)
{
  if (!e || job < 0 || job >= (int)e->jobs.size()) return fail(GD_E_INVALID, "job %d", job);
  if (n < 0 || (n > 0 && (!conf || !mm || !out))) return fail(GD_E_INVALID, "null argument");
  if (precision < GD_PREC_FP32 || precision > GD_PREC_FP64) return fail(GD_E_INVALID, "precision = %d", precision);
  if (n == 0) return GD_OK;
  GD_TRY(set_device(e->device));
  GD_CUDA(cudaStreamSynchronize(e->st));
  return eval_on(e, job, n, conf, mm, precision, out, out64, raw);
}

int gd_ensemble_stats(gd_ensemble_t *e, int job, double *out8)
{
  if (!e || !out8 || job < 0 || job >= (int)e->jobs.size()) return fail(GD_E_INVALID, "job %d", job);
  GD_TRY(set_device(e->device));
  const DevJob &J = e->jobs[job].dj;
  std::vector<RepStats> s(J.nrep);
  GD_CUDA(cudaMemcpyAsync(s.data(), J.stats, sizeof(RepStats) * s.size(), cudaMemcpyDeviceToHost, e->st));
  GD_CUDA(cudaStreamSynchronize(e->st));
  for (int r = 0; r < J.nrep; ++r) {
    const RepStats &x = s[r];
    double *o = out8 + 8 * (size_t)r;
    const double n = (double)x.n_steps;
    o[0] = n;
    o[1] = (double)x.n_accept;
    o[2] = (double)x.n_exch_try;
    o[3] = (double)x.n_exch_acc;
    o[4] = n > 0 ? x.e_sum / n : 0.0;
    o[5] = n > 0 ? std::max(0.0, x.e_sum2 / n - o[4] * o[4]) : 0.0;
    o[6] = x.best_e;
    o[7] = (double)x.best_step;
  }
  return GD_OK;
}

int gd_ensemble_autotune(gd_ensemble_t *e, int steps, char *report, int report_len)
{
  if (!e || steps < 1) return fail(GD_E_INVALID, "autotune: steps = %d", steps);
  if (e->kernel != GD_KERNEL_BATCHED) return GD_OK;
  GD_TRY(set_device(e->device));
  GD_CUDA(cudaStreamSynchronize(e->st));
  // snapshot of everything a Monte Carlo launch writes (records are not written: no record flags)
  std::vector<void *> snaps;
  auto snap_bytes = [](const DevJob &J) {
    return sizeof(ReplicaMC) * (size_t)J.nrep + sizeof(int) * (size_t)J.nrep + sizeof(RepStats) * (size_t)J.nrep;
  };
  int rc = GD_OK;
  for (auto &jb : e->jobs) {
    void *p = nullptr;
    const DevJob &J = jb.dj;
    if (cudaMalloc(&p, snap_bytes(J)) != cudaSuccess) {
      rc = fail(GD_E_NOMEM, "autotune snapshot");
      break;
    }
    unsigned char *b = (unsigned char *)p;
    cudaMemcpyAsync(b, J.rep, sizeof(ReplicaMC) * J.nrep, cudaMemcpyDeviceToDevice, e->st);
    cudaMemcpyAsync(b + sizeof(ReplicaMC) * J.nrep, J.run_acc, sizeof(int) * J.nrep, cudaMemcpyDeviceToDevice, e->st);
    cudaMemcpyAsync(b + (sizeof(ReplicaMC) + sizeof(int)) * J.nrep, J.stats, sizeof(RepStats) * J.nrep,
                    cudaMemcpyDeviceToDevice, e->st);
    snaps.push_back(p);
  }
  auto restore = [&]() {
    for (size_t j = 0; j < e->jobs.size() && j < snaps.size(); ++j) {
      const DevJob &J = e->jobs[j].dj;
      unsigned char *b = (unsigned char *)snaps[j];
      cudaMemcpyAsync(J.rep, b, sizeof(ReplicaMC) * J.nrep, cudaMemcpyDeviceToDevice, e->st);
      cudaMemcpyAsync(J.run_acc, b + sizeof(ReplicaMC) * J.nrep, sizeof(int) * J.nrep, cudaMemcpyDeviceToDevice, e->st);
      cudaMemcpyAsync(J.stats, b + (sizeof(ReplicaMC) + sizeof(int)) * J.nrep, sizeof(RepStats) * J.nrep,
                      cudaMemcpyDeviceToDevice, e->st);
    }
  };
  std::string rep;
  const TileConfig start = e->tc;
  std::vector<std::pair<double, TileConfig>> timed;
  const int shapes[][2] = {{1, 8}, {2, 4}, {2, 8}, {4, 4}, {4, 8}};
  const int warps[] = {4, 6, 8, 10, 12, 14, 16};
  const int group = start.group;  // kept
  const int cluster = start.cluster;  // kept by the candidates of one replica per CTA
  const TileConfig smallest{std::max(4, group), start.kpl, start.ab, 1, group, start.split};
  const bool can_stage = smem_for(e, smallest) <= kSmemLimit;
  int nsm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, e->device);
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  // milliseconds of a launch of shape tc, already configured, by the last of `runs` runs of a strided sample of the work
  // items (heaviest-first order kept), about `waves` waves of the grid, so that a candidate runs the full chunk length
  auto time_shape = [&](const TileConfig &tc, int waves, int runs, const char *what) {
    const int stride = std::max(1, e->n_items / std::max(1, waves * e->grid));
    std::vector<WorkItem> sample;
    for (int i = 0; i < e->n_items; i += stride) sample.push_back(e->h_items[i]);
    WorkItem *d_sample = nullptr;
    if (cudaMalloc(&d_sample, sizeof(WorkItem) * sample.size()) != cudaSuccess ||
        cudaMemcpyAsync(d_sample, sample.data(), sizeof(WorkItem) * sample.size(), cudaMemcpyHostToDevice,
                        e->st) != cudaSuccess) {
      cudaFree(d_sample);
      rc = fail(GD_E_CUDA, "autotune sample");
      return 0.0f;
    }
    KArgs ka = mc_args(e, e->step, steps, 0, nullptr);
    ka.items = d_sample;
    ka.n_items = (int)sample.size();
    float t = 0;
    for (int k = 0; k < runs && rc == GD_OK; ++k) {
      cudaMemsetAsync(e->d_queue, 0, sizeof(int), e->st);
      cudaEventRecord(a, e->st);
      const cudaError_t le = launch_kernel(0, e->precision, e->tc, ka, std::min(e->grid, ka.n_items), e->st);
      cudaEventRecord(b, e->st);
      if (le != cudaSuccess || cudaStreamSynchronize(e->st) != cudaSuccess) rc = fail(GD_E_CUDA, "autotune launch");
      cudaEventElapsedTime(&t, a, b);
      restore();
    }
    cudaFree(d_sample);
    t *= (float)e->n_items / (float)sample.size();   // per whole launch
    char line[160];
    snprintf(line, sizeof line, "%swarps=%d kpl=%d ab=%d stage=%d wide=%d grid=%d items=%d: %.3f ms\n", what,
             tc.warps_per_cta, tc.kpl, tc.ab, tc.stage, tc.wide ? 1 : 0, e->grid, e->n_items, t);
    rep += line;
    return t;
  };
  // the shape that the ensemble has, which the candidates need not contain (its first run warms up for all)
  if (rc == GD_OK) rc = configure(e, start);
  if (rc == GD_OK) timed.emplace_back(time_shape(start, 2, 2, ""), start);
  for (int stage = can_stage ? 1 : 0; stage >= 0; --stage)
  for (const auto &sh : shapes) {
    // FP64 has the shape (1, 8), FP32 the others; a team's kernel has one shape whatever these say
    if ((e->precision == GD_PREC_FP64) != (sh[0] == 1)) continue;
    if (group > 1 && (sh[0] != start.kpl || sh[1] != start.ab)) continue;
    for (int w : warps) {
      if (rc != GD_OK) break;
      // the warps per replica are kept; the candidates are the multiples of it
      if (w % group) continue;
      TileConfig tc{w, sh[0], sh[1], stage, group, start.split, w == group ? cluster : 1};
      // the kernel with more registers by choose_spread's rule
      tc.wide = group == 1 && e->precision != GD_PREC_FP64 && sh[0] == 4 && sh[1] == 8 &&
                (count_items(e, w) + nsm - 1) / nsm * w <= 16;
      if (configure(e, tc) != GD_OK || e->tc.stage != stage) continue;
      timed.emplace_back(time_shape(tc, 2, 1, ""), tc);
    }
  }
  // Two waves rank shapes of uneven jobs no better than to some per cent (512 ligands of 12-64 atoms, 57 waves: three
  // shapes at 1056-1069 ms by their samples take 955, 967 and 990): the present shape and the three fastest others
  // within 5 % of the fastest again on twelve waves.  The present one stays unless another is 1 % faster.
  TileConfig best = start;
  if (rc == GD_OK && timed.size() > 1) {
    std::stable_sort(timed.begin() + 1, timed.end(), [](const auto &x, const auto &y) { return x.first < y.first; });
    const double least = std::min(timed[0].first, timed[1].first);
    size_t n = 1;
    while (n < timed.size() && n < 4 && timed[n].first <= 1.05 * least) ++n;
    timed.resize(n);
    for (auto &c : timed)
      if (rc == GD_OK && (rc = configure(e, c.second)) == GD_OK) c.first = time_shape(c.second, 12, 1, "again: ");
    double best_t = 0.99 * timed[0].first;
    for (size_t k = 1; k < n; ++k)
      if (timed[k].first < best_t) {
        best_t = timed[k].first;
        best = timed[k].second;
      }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaStreamSynchronize(e->st);
  for (void *p : snaps) cudaFree(p);
  e->ev_used = 0;
  e->launches = 0;
  e->all_launches = 0;
  if (rc == GD_OK) rc = configure(e, best);
  char line[160];
  snprintf(line, sizeof line, "chosen: warps=%d kpl=%d ab=%d stage=%d wide=%d\n", best.warps_per_cta, best.kpl, best.ab,
           best.stage, best.wide ? 1 : 0);
  rep += line;
  if (report && report_len > 0) {
    std::strncpy(report, rep.c_str(), (size_t)report_len - 1);
    report[report_len - 1] = 0;
  }
  return rc;
}

// ---------------------------------------------------- checkpoint / resume
namespace {
constexpr uint64_t kSnapMagic = 0x3130504e53444723ull;  // "#GDSNP01"

// Snapshot layout: SnapHeader, then per job a SnapJob, then per job its
// ReplicaMC[nrep], int run_acc[nrep] and RepStats[nrep], in job order.
struct SnapHeader {
  uint64_t magic;
  int32_t njob;
  int32_t step;
};
struct SnapJob {
  int32_t nrep, rid_base;
  uint32_t key0, key1;
};

size_t snap_job_bytes(const DevJob &J)
{
  return (sizeof(ReplicaMC) + sizeof(int) + sizeof(RepStats)) * (size_t)J.nrep;
}
}  // namespace

size_t gd_ensemble_snapshot_bytes(const gd_ensemble_t *e)
{
  if (!e) return 0;
  size_t b = sizeof(SnapHeader) + sizeof(SnapJob) * e->jobs.size();
  for (const auto &j : e->jobs) b += snap_job_bytes(j.dj);
  return b;
}

int gd_ensemble_snapshot(gd_ensemble_t *e, void *buf, size_t bytes)
{
  if (!e || !buf) return fail(GD_E_INVALID, "null argument");
  if (bytes < gd_ensemble_snapshot_bytes(e))
    return fail(GD_E_INVALID, "snapshot buffer of %zu bytes, %zu needed", bytes, gd_ensemble_snapshot_bytes(e));
  GD_TRY(set_device(e->device));
  GD_CUDA(cudaStreamSynchronize(e->st));
  GD_TRY(check_err(e));
  unsigned char *p = (unsigned char *)buf;
  SnapHeader h{kSnapMagic, (int32_t)e->jobs.size(), (int32_t)e->step};
  std::memcpy(p, &h, sizeof h);
  p += sizeof h;
  for (const auto &j : e->jobs) {
    const SnapJob sj{j.dj.nrep, j.dj.rid_base, j.dj.key0, j.dj.key1};
    std::memcpy(p, &sj, sizeof sj);
    p += sizeof sj;
  }
  for (const auto &j : e->jobs) {
    const DevJob &J = j.dj;
    GD_CUDA(cudaMemcpyAsync(p, J.rep, sizeof(ReplicaMC) * J.nrep, cudaMemcpyDeviceToHost, e->st));
    p += sizeof(ReplicaMC) * J.nrep;
    GD_CUDA(cudaMemcpyAsync(p, J.run_acc, sizeof(int) * J.nrep, cudaMemcpyDeviceToHost, e->st));
    p += sizeof(int) * J.nrep;
    GD_CUDA(cudaMemcpyAsync(p, J.stats, sizeof(RepStats) * J.nrep, cudaMemcpyDeviceToHost, e->st));
    p += sizeof(RepStats) * J.nrep;
  }
  GD_CUDA(cudaStreamSynchronize(e->st));
  return GD_OK;
}

int gd_ensemble_restore(gd_ensemble_t *e, const void *buf, size_t bytes)
{
  if (!e || !buf) return fail(GD_E_INVALID, "null argument");
  if (bytes < sizeof(SnapHeader)) return fail(GD_E_INVALID, "snapshot of %zu bytes", bytes);
  const unsigned char *p = (const unsigned char *)buf;
  SnapHeader h;
  std::memcpy(&h, p, sizeof h);
  if (h.magic != kSnapMagic) return fail(GD_E_INVALID, "not an ensemble snapshot");
  if (h.njob != (int32_t)e->jobs.size())
    return fail(GD_E_INVALID, "snapshot of %d jobs, ensemble has %zu", h.njob, e->jobs.size());
  if (bytes < gd_ensemble_snapshot_bytes(e))
    return fail(GD_E_INVALID, "snapshot of %zu bytes, this ensemble's is %zu", bytes, gd_ensemble_snapshot_bytes(e));
  if (h.step < 0) return fail(GD_E_INVALID, "snapshot step %d", h.step);
  p += sizeof h;
  for (size_t k = 0; k < e->jobs.size(); ++k) {
    SnapJob sj;
    std::memcpy(&sj, p, sizeof sj);
    p += sizeof sj;
    const DevJob &J = e->jobs[k].dj;
    // the Philox draws are keyed by (seed, replica, step): a snapshot continues
    // bit for bit only in an ensemble of the same replicas and seeds
    if (sj.nrep != J.nrep || sj.rid_base != J.rid_base || sj.key0 != J.key0 || sj.key1 != J.key1)
      return fail(GD_E_INVALID, "snapshot job %zu: replicas/seed differ from the ensemble's", k);
  }
  GD_TRY(set_device(e->device));
  GD_CUDA(cudaStreamSynchronize(e->st));
  for (const auto &j : e->jobs) {
    const DevJob &J = j.dj;
    GD_CUDA(cudaMemcpyAsync(J.rep, p, sizeof(ReplicaMC) * J.nrep, cudaMemcpyHostToDevice, e->st));
    p += sizeof(ReplicaMC) * J.nrep;
    GD_CUDA(cudaMemcpyAsync(J.run_acc, p, sizeof(int) * J.nrep, cudaMemcpyHostToDevice, e->st));
    p += sizeof(int) * J.nrep;
    GD_CUDA(cudaMemcpyAsync(J.stats, p, sizeof(RepStats) * J.nrep, cudaMemcpyHostToDevice, e->st));
    p += sizeof(RepStats) * J.nrep;
  }
  GD_CUDA(cudaStreamSynchronize(e->st));
  e->step = h.step;
  return GD_OK;
}

int gd_ensemble_destroy(gd_ensemble_t *e)
{
  destroy(e);
  return GD_OK;
}

}  // extern "C"

// ------------------------------------------------------------- layout --
// Sizes and offsets of the boundary structs, for bindings that mirror them.
extern "C" long long gd_layout(const char *what)
{
  if (!what) return -1;
  const std::string w(what);
#define GD_L(name, expr) \
  if (w == name) return (long long)(expr);
  GD_L("sizeof.Complex", sizeof(Complex))
  GD_L("sizeof.Record", sizeof(Record))
  GD_L("sizeof.ReplicaMC", sizeof(ReplicaMC))
  GD_L("sizeof.EnePara", sizeof(EnePara))
  GD_L("sizeof.EnePara0", sizeof(EnePara0))
  GD_L("sizeof.Ligand", sizeof(Ligand))
  GD_L("sizeof.Protein", sizeof(Protein))
  GD_L("sizeof.Kde", sizeof(Kde))
  GD_L("sizeof.Mcs", sizeof(Mcs))
  GD_L("sizeof.ParaT", sizeof(ParaT))
  GD_L("Complex.lig", offsetof(Complex, lig))
  GD_L("Complex.prt", offsetof(Complex, prt))
  GD_L("Complex.psp", offsetof(Complex, psp))
  GD_L("Complex.kde", offsetof(Complex, kde))
  GD_L("Complex.mcs", offsetof(Complex, mcs))
  GD_L("Complex.enepara", offsetof(Complex, enepara))
  GD_L("Complex.temp", offsetof(Complex, temp))
  GD_L("Complex.replica", offsetof(Complex, replica))
  GD_L("Complex.size", offsetof(Complex, size))
  GD_L("Complex.mcpara", offsetof(Complex, mcpara))
  GD_L("Complex.lig_file", offsetof(Complex, lig_file))
  GD_L("Complex.rep_begin", offsetof(Complex, rep_begin))
  GD_L("Complex.rep_end", offsetof(Complex, rep_end))
  GD_L("Complex.signal", offsetof(Complex, signal))
  GD_L("EnePara.w", offsetof(EnePara, w))
  GD_L("EnePara.hpl0", offsetof(EnePara, hpl0))
  GD_L("EnePara.kde2", offsetof(EnePara, kde2))
  GD_L("Record.next_entry", offsetof(Record, next_entry))
  GD_L("sizeof.gd_job_desc_t", sizeof(gd_job_desc_t))
  GD_L("sizeof.gd_pocket_desc_t", sizeof(gd_pocket_desc_t))
  GD_L("sizeof.gd_server_config_t", sizeof(gd_server_config_t))
  GD_L("sizeof.gd_request_t", sizeof(gd_request_t))
  GD_L("sizeof.gd_result_t", sizeof(gd_result_t))
  GD_L("sizeof.gd_server_stats_t", sizeof(gd_server_stats_t))
  GD_L("sizeof.gd_load_args_t", sizeof(gd_load_args_t))
  GD_L("sizeof.gd_cluster_t", sizeof(gd_cluster_t))
  GD_L("gd_server_stats_t.warps_per_cta", offsetof(gd_server_stats_t, warps_per_cta))
  GD_L("gd_result_t.t_done", offsetof(gd_result_t, t_done))
#undef GD_L
  return -1;
}

// ------------------------------------------------------ force field --
// OptimizeEnepara (src/frontend/util_optimize_soa.C:489-540): the same float
// operations in the same order, so the tables match the reference bit for bit.
extern "C" int gd_optimize_enepara(const EnePara0 *e0, EnePara *e)
{
  if (!e0 || !e) return fail(GD_E_INVALID, "null argument");
  std::memset(e, 0, sizeof(EnePara));
  const float sqrt_2_pi = sqrtf(2.0f * 3.1415926535f);
  for (int i = 0; i < GD_MAXTP2; ++i)
    for (int j = 0; j < GD_MAXTP1; ++j) {
      const float tmp = e0->vdw[j][i][0] * e0->lj[2];
      e->p1a[i][j] = 2.0f * e0->vdw[j][i][1] * powf(tmp, 9.0f);
      e->p2a[i][j] = 3.0f * e0->vdw[j][i][1] * powf(tmp, 6.0f);
    }
  e->lj0 = e0->lj[0];
  e->lj1 = e0->lj[1];
  e->el1 = e0->el[1];
  e->el0 = e0->el[0];
  e->a1 = 4.0f - 3.0f * e0->el[0];
  e->b1 = 2.0f * e0->el[0] - 3.0f;
  for (int i = 0; i < GD_MAXTP2; ++i)
    for (int j = 0; j < GD_MAXTP1; ++j) {
      e->pmf0[i][j] = e0->pmf[j][i][0];
      e->pmf1[i][j] = e0->pmf[j][i][1];
      e->hdb0[i][j] = e0->hdb[j][i][0];
      e->hdb1[i][j] = 1.0f / e0->hdb[j][i][1];
    }
  for (int i = 0; i < GD_MAXTP4; ++i) e->hpp[i] = e0->hpp[i];
  for (int i = 0; i < GD_MAXTP2; ++i) {
    e->hpl0[i] = e0->hpl[i][0];
    e->hpl1[i] = e0->hpl[i][1];
    e->hpl2[i] = logf(1.0f / (e->hpl1[i] * sqrt_2_pi));
  }
  e->kde2 = -0.5f / (e0->kde * e0->kde);
  e->kde3 = powf(e0->kde * sqrt_2_pi, 3.0f);
  for (int i = 0; i < GD_MAXWEI; ++i) {
    e->w[i] = e0->w[i];
    e->a_para[i] = e0->a_para[i];
    e->b_para[i] = e0->b_para[i];
  }
  return GD_OK;
}

// ------------------------------------------------------------ timing --
extern "C" void *gd_ensemble_stream(const gd_ensemble_t *e) { return e ? (void *)e->st : nullptr; }

namespace {
// Independent FMA chains: 8 accumulators per thread so the FMA pipe, not
// latency, bounds the loop; the result is stored so nothing is dead code.
__global__ void fma_peak_kernel(float *out, int iters, float a, float b)
{
  float x0 = threadIdx.x * 1e-3f, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6,
        x7 = x0 + 7;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      x0 = fmaf(x0, a, b); x1 = fmaf(x1, a, b); x2 = fmaf(x2, a, b); x3 = fmaf(x3, a, b);
      x4 = fmaf(x4, a, b); x5 = fmaf(x5, a, b); x6 = fmaf(x6, a, b); x7 = fmaf(x7, a, b);
    }
  }
  out[blockIdx.x * blockDim.x + threadIdx.x] = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
}
}  // namespace

// Measured FP32 FMA throughput of the current device in TFLOP/s (2 flops per FMA).
extern "C" int gd_fp32_peak(double *tflops)
{
  if (!tflops) return fail(GD_E_INVALID, "null argument");
  int dev = 0, nsm = 0;
  GD_CUDA(cudaGetDevice(&dev));
  GD_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int threads = 512, blocks = nsm * 4, iters = 4096;
  float *out = nullptr;
  GD_CUDA(cudaMalloc(&out, sizeof(float) * threads * blocks));
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  fma_peak_kernel<<<blocks, threads>>>(out, 64, 0.999f, 1e-3f);  // warm-up
  cudaEventRecord(a);
  fma_peak_kernel<<<blocks, threads>>>(out, iters, 0.999f, 1e-3f);
  cudaEventRecord(b);
  const cudaError_t e = cudaEventSynchronize(b);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(out);
  if (e != cudaSuccess) return fail(GD_E_CUDA, "gd_fp32_peak: %s", cudaGetErrorString(e));
  const double flops = 2.0 * 8.0 * 16.0 * (double)iters * threads * blocks;
  *tflops = flops / (ms * 1e-3) / 1e12;
  return GD_OK;
}
