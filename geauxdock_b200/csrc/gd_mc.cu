// gd_mc.cu -- the batched Monte Carlo kernel (one warp per replica), the
// pose-evaluation kernel that shares its energy code, and the replica
// exchange kernels.
//
// Mapping to the hardware.  The reference runs one 1024-thread block per
// replica and synchronises the block six or more times per step
// (src/backend_gpu/kernel_cuda_l1_montecarlo.cu:284-527).  Here one warp owns
// one replica for a whole chunk of steps: the step needs no block barrier,
// only warp shuffles.  A CTA holds R replica-warps that share one protein
// conformation; per work item the CTA stages the force-field parameters (when it
// pays, also the conformation itself) into shared
// memory with 1-D bulk (TMA) copies, and its replica-warps read them every
// step.  A persistent grid takes work items from an atomic queue, heaviest
// first.
//
// Pair loop, pass 1 (every term but the hydrophobic contact).  Lane i holds
// pocket points row+i+32j (j < KPL) in registers.  The FP32 ligand sits in
// shared memory as atom pairs, and with KPL even every add, multiply and FMA
// evaluates atoms 2k and 2k+1 against one point as one packed f32x2
// instruction (sm_100).  Per work item the CTA builds from the per-type tables
// one entry per (atom pair, point type) with the two atoms' values interleaved,
// so the loop walks atom pairs with no grouping by atom type; the sparse
// hydrogen-bond term is evaluated only for the atom pairs where some point of
// the row needs it, and the pocket-specific term is walked after the loop over
// the potential's non-zero cells of the conformation.  In FP64 the atoms are
// walked one type group at a time in scalar arithmetic.  Pass 2
// (the hydrophobic contact) visits only the rows holding cdc == 1 points, packed
// over atom pairs the same way, and keeps per-atom sums in registers for AB
// atoms at a time.
//
// Arithmetic follows src/backend_gpu/energy_prt_v1.cu:8-174 term by term, in
// rearranged FP32 forms derived in the comments; the special functions use
// the single-instruction PTX approximations (rsqrt/rcp/ex2.approx).  The
// FP32-Kahan variant (the default) adds each row's partial sums of the three
// dense terms into the lane totals with compensated summation and reduces
// across lanes with a compensated butterfly; the FP64 variant evaluates the same
// rearrangement of the Lennard-Jones term and the other terms as they stand in
// double, with special functions of its own (gd_energy.cuh).
#include <algorithm>
#include <cstdio>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <utility>

#include "gd_device.cuh"
#include "gd_internal.h"
#include "gd_pack.h"

namespace gd {

namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kSqrt2PiInvNeg = -0.3989422804014327f;  // -1/sqrt(2 pi), kernel_cuda_l1_montecarlo.cu:14
constexpr double kSqrt2PiInvNegD = -0.39894228040143267794;  // the same in FP64
// bound of the staging waits when the wait_limit option is 0: one second
constexpr uint64_t kWaitLimitNs = 1000000000ull;

__device__ __forceinline__ uint64_t wait_limit_ns(uint32_t us) { return us ? 1000ull * us : kWaitLimitNs; }

template <typename T>
struct alignas(16) V4 {
  T x, y, z, w;
};

// FP32 ligand in shared memory as atom pairs: component k of each float2 is
// atom 2i + k of pair i, so that packed f32x2 arithmetic reads two atoms as one
// register pair.  An odd atom count ends with an inert dummy half.
struct alignas(16) LigPair {
  float2 x, y, z, q;
};
__device__ __forceinline__ V4<float> atom_at(const LigPair *lig, int a)
{
  const float *f = reinterpret_cast<const float *>(lig + (a >> 1)) + (a & 1);
  return V4<float>{f[0], f[2], f[4], f[6]};
}
__device__ __forceinline__ V4<double> atom_at(const V4<double> *lig, int a) { return lig[a]; }

__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

}  // namespace

// Bounds checks of the debug build (-DGD_CHECK, libgdock_check.so): every
// instrumented index is compared with the length of its array; one out of
// range records (site, index, length) in g_check once and is replaced by 0,
// so the access stays inside the array and the run goes on.  gd_check_report
// reads the record.  In the product build GD_AT(i, n, site) is the tokens of i.
#ifdef GD_CHECK
static __device__ int g_check[4];
__device__ __forceinline__ long long check_at(long long i, long long n, int site)
{
  if (i >= 0 && i < n) return i;
  if (atomicCAS(&g_check[0], 0, 1) == 0) {
    g_check[1] = site;
    g_check[2] = (int)i;
    g_check[3] = (int)n;
  }
  return 0;
}
#define GD_AT(i, n, site) ::gd::check_at((long long)(i), (long long)(n), (site))
#define GD_CHECK_ARG(...) , __VA_ARGS__
#else
// unparenthesised on purpose: the index expression keeps its own grouping
// (a pointer plus an index sum is then computed as written), so that the
// product build compiles to exactly the code without the checks.  A use
// inside a product or another operator must parenthesise its argument
// (2 * GD_AT((k + m), ...)), or it would expand to 2 * k + m.
#define GD_AT(i, n, site) i
#define GD_CHECK_ARG(...)
#endif
// sites reported by gd_check_report
enum CheckSite { kSiteLig = 1, kSiteApt, kSiteAph, kSiteAhd, kSitePos, kSitePsp, kSiteKde, kSiteMcs, kSiteLgrp,
                 kSiteTcc, kSiteLigConf, kSitePrtConf, kSiteRep, kSiteTmp, kSiteTab = 16 };

}  // namespace gd

#include "gd_energy.cuh"

namespace gd {

// ----------------------------------------------------------- smem layout --
struct SmemLayout {
  uint32_t params, lgrp, pos, aux, apt, aph, ahd, warp0, warp_bytes, lig_bytes, total;
  uint32_t team0, team_bytes, parts;  // teams of warps (gd_team.cuh)
};

__host__ __device__ inline uint32_t align16(uint32_t x) { return (x + 15u) & ~15u; }

constexpr int kDrawSteps = 16;  // Monte Carlo steps whose random numbers a warp of a team draws at once
// 32-point chunks of each of the KDE and pocket-specific walks whose terms a team of 8 or more warps keeps in shared
// memory; a smaller team gives each walk to one warp
__host__ __device__ inline int team_chunks(int G) { return G >= 8 ? 24 : 0; }

// Values per lane and row that pass 1 leaves in shared memory, times 32: four sums, or in the one-warp order of a
// team of 8 or more warps the two components' seven (HalfRow).
__host__ __device__ inline int team_row_reals(int G, int V, bool fp64) { return G >= 8 && V == 1 && !fp64 ? 448 : 128; }

// Points of a pass 1 row, the unit a team deals out: the one-warp kernel's, or with the split order (V > 1) half.
__host__ __device__ inline int team_row(int V) { return V > 1 ? kHalfPoints : kRowPoints; }

// P: points staged (0: none); Pall: points of the largest conformation.
__host__ __device__ inline SmemLayout smem_layout(int P, int Pall, int lig_slots, int warps, bool fp64, int group = 1,
                                                   int split = 1)
{
  SmemLayout s;
  uint32_t off = 0;
  s.params = off;  // the scalar prefix of DevParams
  off = align16(off + (uint32_t)kParamScalarBytes);
  s.lgrp = off;
  off = align16(off + (uint32_t)sizeof(int2) * kMaxAtoms);
  s.pos = off;
  off = align16(off + 16u * (uint32_t)P);
  s.aux = off;
  off = align16(off + 8u * (uint32_t)P);
  // FP32: per (atom pair, point type) tables of the atom-pair pair loop and a header per pair; FP64: per (type group,
  // point type), and the exponential's table in the place of the headers
  const uint32_t npairs = (uint32_t)(lig_slots + 1) / 2u;
  const uint32_t entries = (uint32_t)kTabCols * (fp64 ? (uint32_t)(lig_slots < kLigTypes ? lig_slots : kLigTypes) : npairs);
  s.apt = off;
  off = align16(off + (fp64 ? 16u : 32u) * entries);
  s.aph = off;
  off = align16(off + 16u * entries);
  s.ahd = off;
  off = align16(off + (fp64 ? 16u * (uint32_t)kExpTab : 16u * npairs));
  s.lig_bytes = (uint32_t)lig_slots * (fp64 ? 32u : 16u);  // V4<double> per atom, or LigPair per two atoms
  // per replica: ReplicaMC state, EnergyScratch (192 B), WarpStats (64 B); per warp the rotated ligand
  const uint32_t state = (uint32_t)sizeof(ReplicaMC) + 192u + 64u;
  s.team0 = off;
  s.team_bytes = 0;
  s.parts = 0;
  if (group > 1) {
    // per team: the state, the rows' sums per lane, the contact sums per atom and share of the split order, the
    // walks' terms (chunks) or sums per lane
    const uint32_t real = fp64 ? 8u : 4u, V = (uint32_t)split;
    const uint32_t walk = 64u * (V > 1 ? 0u : (uint32_t)team_chunks(group)) + 32u * V;
    s.parts = (uint32_t)sizeof(ReplicaMC) + 64u + real * 84u;
    s.team_bytes = align16(s.parts + real * ((uint32_t)team_row_reals(group, split, fp64) * (uint32_t)(Pall / team_row(split)) + V * (uint32_t)kMaxAtoms + 2u * walk));
    off += s.team_bytes * (uint32_t)(warps / group);
  }
  s.warp_bytes = align16(s.lig_bytes + (group > 1 ? (uint32_t)kDrawSteps * 40u : state));
  s.warp0 = off;
  off += s.warp_bytes * (uint32_t)warps;
  s.total = off;
  return s;
}

// Per-warp results of energy_warp, and the pose it is given.
struct EnergyScratch {
  double e[10];    // normalised terms and total
  double raw[9];   // terms before the per-atom division and normalisation
  float mm[6];     // pose being evaluated (input)
  float pad_[4];
};
static_assert(sizeof(EnergyScratch) == 192, "EnergyScratch size is part of the smem layout");

// ------------------------------------------------------------- energy --
// Energy of ligand conformation ilig at pose out->mm in protein conformation
// iprt, by one warp; writes e[0..9] (normalised terms and total) and raw[0..8].
template <int PREC, int KPL, int AB, bool C4>
__device__ __noinline__ void energy_warp(const DevJob &J, const DevParams *__restrict__ par,
                                         const float4 *__restrict__ pos, const float2 *__restrict__ aux,
                                         const int2 *__restrict__ lgrp, const float4 *__restrict__ apt,
                                         const float4 *__restrict__ aph, const int4 *__restrict__ ahd, void *ligbuf,
                                         int ilig, int iprt, EnergyScratch *out)
{
  using T = RealOf<PREC>;
  const int lane = lane_id();
  const int L = J.natom, P = J.npoint_pad;
  LigOf<PREC> *lig = reinterpret_cast<LigOf<PREC> *>(ligbuf);
  rotate_ligand<PREC>(J, ilig, lane < 6 ? out->mm[lane] : 0.0f, lig);

  // pass 1, row by row
  RowSums<PREC> rs;
  if constexpr (PREC == kFP64) {
    for (int row = 0; row < P; row += kRowPoints) {
      double h[4];
      pass1_row64(lig, L, lgrp, par, reinterpret_cast<const double2 *>(apt), aph, reinterpret_cast<const double *>(ahd), row,
                  P, pos, aux, h);
#pragma unroll
      for (int t = 0; t < 4; ++t) rs.add(t, h[t]);
    }
  } else {
    const PairConst kc = PairConst::load(par);
    for (int row = 0; row < P; row += 32 * KPL) {
      const float4 r = pass1_row<KPL, false>(lig, (L + 1) >> 1, row, P, pos, aux, apt, aph, ahd, kc);
      rs.add(0, r.x);
      rs.add(1, r.y);
      rs.add(2, r.z);
      rs.add(3, r.w);
    }
  }
  const T s_psp = psp_walk<PREC, C4>(J, iprt, lig, 0, 1);

  // pass 2: one lane per atom applies the restraint
  T ehpc = 0;
  {
    const int rows = contact_rows(J, iprt);
    for (int a0 = 0; a0 < L; a0 += AB) {
      const T S = contact_block<PREC, AB>(lig, L, a0, 0, kHalfPoints, rows, pos, aux, P);
      const int a = a0 + lane / (32 / AB);
      if (a < L && (lane & (32 / AB - 1)) == 0) ehpc = add_(ehpc, contact_restraint(par, lgrp, a, L, S));
    }
    ehpc = warp_sum(ehpc);
  }

  const T vdw = rs.total(0), ele = rs.total(1), pmf = rs.total(2), psp = warp_sum(s_psp), hdb = rs.total(3);
  const T ekde = warp_sum(kde_walk<PREC>(J, par, lig, 0, 1));
  const T elhm = mcs_sums<PREC>(J, lig, 1, nullptr);
  const T dst = centre_dist2<T>(J, ilig, iprt, lane < 6 ? out->mm[lane] : 0.0f);

  // lane i finishes term i; the weighted total in term order
  T x = dst;
  x = lane == 0 ? vdw : x;
  x = lane == 1 ? ele : x;
  x = lane == 2 ? pmf : x;
  x = lane == 3 ? psp : x;
  x = lane == 4 ? hdb : x;
  x = lane == 5 ? ehpc : x;
  x = lane == 6 ? ekde : x;
  x = lane == 7 ? elhm : x;
  const int term = lane < 9 ? lane : 8;
  const T raw = raw_term<PREC>(term, scaled_sum<PREC>(term, x, par), J.nmcs);
  const T v = norm_term(term, raw, par, L);
  T tot = 0;
#pragma unroll
  for (int i = 0; i < 9; ++i) tot = fma_((T)par->w[i], __shfl_sync(0xffffffffu, v, i), tot);
  if (lane < 9) {
    out->raw[lane] = (double)raw;
    out->e[lane] = (double)v;
  }
  if (lane == 9) out->e[9] = (double)tot;
  __syncwarp();
}

// ------------------------------------------------------------ kernels --

// Stage the shared data of work item `wi` into shared memory.  Returns false,
// in every thread of the CTA alike, if the bulk copies did not complete within
// the wait limit; the barrier phase is then left open (see stage_abandon).
__device__ bool stage_item(const KArgs &A, const DevJob &J, const WorkItem &wi, unsigned char *smem,
                           const SmemLayout &sl, uint64_t *bar, uint32_t &phase)
{
  const int P = J.npoint_pad;
  const bool pocket_in_smem = A.P > 0;
  if (threadIdx.x == 0) {
    fence_proxy_async_smem();
    const uint32_t pbytes = (uint32_t)kParamScalarBytes;
    mbar_expect_tx(bar, pbytes + (pocket_in_smem ? 24u * (uint32_t)P : 0u) + A.stall_bytes);
    bulk_g2s(smem + sl.params, J.par, pbytes, bar);
    if (pocket_in_smem) {
      bulk_g2s(smem + sl.pos, J.pos + (size_t)wi.prt * P, 16u * (uint32_t)P, bar);
      bulk_g2s(smem + sl.aux, J.aux + (size_t)wi.prt * P, 8u * (uint32_t)P, bar);
    }
  }
  int2 *lg = reinterpret_cast<int2 *>(smem + sl.lgrp);
  for (int a = threadIdx.x; a < J.natom; a += blockDim.x) lg[a] = J.lgrp[a];
  // one decision for the whole CTA: a thread that saw the phase complete and
  // one that gave up must not go separate ways
  const bool ok = __syncthreads_and(mbar_wait(bar, phase, wait_limit_ns(A.wait_limit)) ? 1 : 0) != 0;
  phase ^= 1u;
  return ok;
}

// After stage_item gave up: before the CTA returns (and its shared memory goes
// to another CTA), let the copies it issued land.  Bytes the test hook
// announced without a copy are taken off the barrier first, so that the phase
// completes exactly when the real copies have arrived; the wait is bounded
// again.  `phase` is the parity stage_item already advanced.
__device__ void stage_abandon(const KArgs &A, uint64_t *bar, uint32_t phase)
{
  if (threadIdx.x == 0 && A.stall_bytes) mbar_complete_tx(bar, A.stall_bytes);
  __syncthreads();
  (void)__syncthreads_and(mbar_wait(bar, phase ^ 1u, wait_limit_ns(A.wait_limit)) ? 1 : 0);
}

// The shared data of work item `wi`: staged, and its pair tables built, where the
// CTA's previous item had another job or protein conformation.  Returns false
// in every thread alike after a wait gave up (the kernel then returns).
template <int PREC>
__device__ bool load_item(const KArgs &A, const DevJob &J, const WorkItem &wi, unsigned char *smem,
                          const SmemLayout &sl, uint64_t *bar, uint32_t &phase, int &prev_job, int &prev_prt)
{
  if (wi.job != prev_job || wi.prt != prev_prt) {
    if (!stage_item(A, J, wi, smem, sl, bar, phase)) {
      if (threadIdx.x == 0) atomicOr(A.err, kErrTimeout);
      stage_abandon(A, bar, phase);
      return false;
    }
    __syncthreads();  // type groups are in shared memory
    if (wi.job != prev_job) {
      const int2 *lg = reinterpret_cast<const int2 *>(smem + sl.lgrp);
      if constexpr (PREC == kFP64)
        build_pair_tables64(J, lg, reinterpret_cast<double2 *>(smem + sl.apt), reinterpret_cast<float4 *>(smem + sl.aph),
                            reinterpret_cast<double *>(smem + sl.ahd));
      else
        build_pair_tables(J.natom, J.par, lg, reinterpret_cast<float4 *>(smem + sl.apt),
                          reinterpret_cast<float4 *>(smem + sl.aph), reinterpret_cast<int4 *>(smem + sl.ahd));
    }
    prev_job = wi.job;
    prev_prt = wi.prt;
    __syncthreads();
  }
  return true;
}

// The next work item's index: from the queue, or (mode 2, no item list) the CTA's
// turn; and the item.  Mode 2 poses of one CTA may have any protein conformation:
// nothing of a conformation is staged, and after the first turn nothing is shared
// between a CTA's warps (or teams) that a turn writes.
template <int MODE>
__device__ __forceinline__ int next_item(const KArgs &A, int turn, int *s_item)
{
  if constexpr (MODE == 2) return blockIdx.x + turn * gridDim.x;
  if (threadIdx.x == 0) *s_item = atomicAdd(A.queue, 1);
  __syncthreads();
  return *s_item;
}
template <int MODE>
__device__ __forceinline__ WorkItem work_item(const KArgs &A, int it, int R)
{
  if constexpr (MODE == 2) return WorkItem{0, 0, it * R, min(R, A.n_poses - it * R)};
  return A.items[it];
}

// Mode 2: a pose whose conformations are out of range gets NaN and the error flag.
__device__ __forceinline__ bool bad_pose(const KArgs &A, const DevJob &J, int r, int ilig, int iprt, bool tell)
{
  if (ilig >= 0 && ilig < J.nlig && iprt >= 0 && iprt < J.nprt) return false;
  if (tell && lane_id() < 10) A.out[10 * (size_t)r + lane_id()] = __int_as_float(0x7fc00000);
  if (tell && lane_id() == 0) atomicOr(A.err, kErrSize);
  return true;
}

// Per-replica FP64 statistics kept in shared memory during a chunk (one lane).
struct WarpStats {
  double e_sum, e_sum2, best_e;
  long long n_acc;
  float best_mm[6];
  int best_step;
  int pad_;
};

__device__ __forceinline__ void load_stats(WarpStats *w, const RepStats &S)
{
  w->e_sum = 0.0;
  w->e_sum2 = 0.0;
  w->n_acc = 0;
  w->best_e = S.best_e;
  w->best_step = S.best_step;
  for (int i = 0; i < 6; ++i) w->best_mm[i] = S.best_mm[i];
}

// Step s ended with total energy ecur at pose mm.
__device__ __forceinline__ void step_stats(WarpStats *w, int accept, double ecur, int s, const float *mm)
{
  w->n_acc += accept;
  w->e_sum += ecur;
  w->e_sum2 = fma_(ecur, ecur, w->e_sum2);
  if (w->best_step < 0 || ecur < w->best_e) {
    w->best_e = ecur;
    w->best_step = s;
    for (int i = 0; i < 6; ++i) w->best_mm[i] = mm[i];
  }
}

__device__ __forceinline__ void store_stats(RepStats &S, const WarpStats *w, int nsteps)
{
  S.e_sum += w->e_sum;
  S.e_sum2 += w->e_sum2;
  S.n_steps += nsteps;
  S.n_accept += w->n_acc;
  S.best_e = w->best_e;
  S.best_step = w->best_step;
  for (int i = 0; i < 6; ++i) S.best_mm[i] = w->best_mm[i];
}

// 80 registers keep 24 warps on an SM.  WIDE, for launches that have 16 or fewer for each: with 128 the points of a row
// overlap further, which counts where few warps hide each other's latency (80 atoms x 2200 points, a step beside 8 and
// 16 warps per SM 402 -> 353 us and 570 -> 543 us).
template <int MODE, int PREC, int KPL, int AB, bool WIDE = false>
__global__ void __maxnreg__(PREC == kFP64 || WIDE ? 128 : 80) mc_kernel(KArgs A)
{
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int s_item;
  const SmemLayout sl = smem_layout(A.P, A.Pall, A.lig_slots, blockDim.x / 32, PREC == kFP64);
  const int warp = threadIdx.x >> 5;
  const int lane = lane_id();
  // a Complex the device packer refused (gd_devpack.cu) leaves its job unread
  if (*(volatile int *)A.err & kErrPack) return;
  if (threadIdx.x == 0) mbar_init(&bar, 1);
  __syncthreads();
  uint32_t phase = 0;
  int prev_job = -1, prev_prt = -1;

  for (int turn = 0;; ++turn) {
    const int it = next_item<MODE>(A, turn, &s_item);
    if (it >= A.n_items) break;
    const WorkItem wi = work_item<MODE>(A, it, blockDim.x >> 5);
    const DevJob &J = A.jobs[wi.job];
    if (!load_item<PREC>(A, J, wi, smem, sl, &bar, phase, prev_job, prev_prt)) return;
    const float4 *apt = reinterpret_cast<const float4 *>(smem + sl.apt);
    const float4 *aph = reinterpret_cast<const float4 *>(smem + sl.aph);
    const int4 *ahd = reinterpret_cast<const int4 *>(smem + sl.ahd);

    const DevParams *par = reinterpret_cast<const DevParams *>(smem + sl.params);  // its scalar prefix
    // the protein conformation: staged in shared memory, or read through L1
    const float4 *pos = A.P > 0 ? reinterpret_cast<const float4 *>(smem + sl.pos)
                                : J.pos + (size_t)wi.prt * J.npoint_pad;
    const float2 *aux = A.P > 0 ? reinterpret_cast<const float2 *>(smem + sl.aux)
                                : J.aux + (size_t)wi.prt * J.npoint_pad;
    const int2 *lgrp = reinterpret_cast<const int2 *>(smem + sl.lgrp);
    unsigned char *wbase = smem + sl.warp0 + (size_t)warp * sl.warp_bytes;
    void *ligbuf = wbase;
    ReplicaMC *srep = reinterpret_cast<ReplicaMC *>(wbase + sl.lig_bytes);
    EnergyScratch *esc = reinterpret_cast<EnergyScratch *>(wbase + sl.lig_bytes + sizeof(ReplicaMC));
    WarpStats *wst = reinterpret_cast<WarpStats *>(wbase + sl.lig_bytes + sizeof(ReplicaMC) + sizeof(EnergyScratch));

    if (warp < wi.count) {
      const int r = wi.rep0 + warp;  // job-local index
      if constexpr (MODE >= 1) {
        // ---- pose evaluation
        const int ilig = A.conf[2 * (size_t)r], iprt = A.conf[2 * (size_t)r + 1];
        if constexpr (MODE == 2) {
          if (bad_pose(A, J, r, ilig, iprt, true)) continue;  // no barrier follows in this mode
          pos = J.pos + (size_t)iprt * J.npoint_pad;
          aux = J.aux + (size_t)iprt * J.npoint_pad;
        }
        if (lane < 6) esc->mm[lane] = A.mm[6 * (size_t)r + lane];
        __syncwarp();
        energy_warp<PREC, KPL, AB, MODE == 2>(J, par, pos, aux, lgrp, apt, aph, ahd, ligbuf, ilig, iprt, esc);
        if (lane < 10) {
          A.out[10 * (size_t)r + lane] = (float)esc->e[lane];
          if (A.out64) A.out64[10 * (size_t)r + lane] = esc->e[lane];
        }
        if (A.raw && lane < 9) A.raw[9 * (size_t)r + lane] = (float)esc->raw[lane];
        __syncwarp();
      } else {
        // ---- Monte Carlo chunk for replica r
        const int gr = J.rid_base + r;
        int *sw = reinterpret_cast<int *>(srep);
        sw[lane] = reinterpret_cast<const int *>(J.rep + GD_AT(r, J.nrep, kSiteRep))[lane];
        if (lane == 0) load_stats(wst, J.stats[r]);
        __syncwarp();
        int acc = J.run_acc[r];
        const int ilig = srep->idx_lig, iprt = srep->idx_prt;
        const double mbeta = (double)J.minus_beta[GD_AT(srep->idx_tmp, J.ntmp, kSiteTmp)];
        Record *rec = (J.rec && (A.flags & kMcRecord)) ? J.rec + r : nullptr;
        int ne = 0;
        if (J.rec && (A.flags & kMcResetRecord)) {
          if (lane == 0) J.rec[r].next_entry = 0;
        } else if (rec) {
          ne = rec->next_entry;
        }
        const bool initial = (A.flags & kMcInitial) != 0;

        const int s0 = (A.d_step ? *A.d_step + A.s_begin : A.s_begin) + J.step0;
        const int nsteps = J.nsteps > 0 ? min(J.nsteps, A.nsteps) : A.nsteps;
        for (int s = s0; s < s0 + nsteps; ++s) {
          if (acc) {
            // record the old state, kernel_cuda_l1_montecarlo.cu:290-297
            if (lane == 0) srep->step = s;
            __syncwarp();
            if (rec && ne < GD_STEPS_PER_DUMP) reinterpret_cast<int *>(&rec->replica[ne])[lane] = sw[lane];
            ++ne;
          }
          // draws of step s: counter {s, replica, 0, 0} -> move x y z, rot x;
          // {s, replica, 0, 1} -> rot y z, accept (lane 0 and lane 1 compute one each)
          float u_acc = 0.0f;
          if (!initial) {
            const Philox4 d = philox4x32_10((uint32_t)s, (uint32_t)gr, 0u, (uint32_t)(lane & 1), J.key0, J.key1);
            float u[7];
#pragma unroll
            for (int k = 0; k < 4; ++k) u[k] = u01(__shfl_sync(0xffffffffu, d.v[k], 0));
#pragma unroll
            for (int k = 4; k < 7; ++k) u[k] = u01(__shfl_sync(0xffffffffu, d.v[k - 4], 1));
            u_acc = u[6];
            if (lane < 6) {
              float v = u[0];
#pragma unroll
              for (int i = 1; i < 6; ++i) v = (lane == i) ? u[i] : v;
              esc->mm[lane] = __fmaf_rn(par->move_scale[lane], v, srep->movematrix[lane]);
            }
          } else if (lane < 6) {
            esc->mm[lane] = __fmaf_rn(par->move_scale[lane], 0.0f, srep->movematrix[lane]);
          }
          __syncwarp();
          energy_warp<PREC, KPL, AB, false>(J, par, pos, aux, lgrp, apt, aph, ahd, ligbuf, ilig, iprt, esc);
          const float etot = (float)esc->e[9];

          // Metropolis test in FP64, kernel_cuda_l1_montecarlo.cu:485-507
          int accept = 1;
          if (!initial) {
            const double lr = ((double)etot - (double)srep->energy[9]) * mbeta;
            accept = log((double)u_acc) < lr;
          }
          __syncwarp();
          if (accept) {
            if (lane < 10) srep->energy[lane] = (float)esc->e[lane];
            if (lane < 6) srep->movematrix[lane] = esc->mm[lane];
          }
          __syncwarp();
          if (lane == 0) step_stats(wst, accept, (double)srep->energy[9], s, srep->movematrix);
          acc = accept;
        }

        if (lane == 0) {
          J.run_acc[r] = acc;
          if (A.flags & kMcStoreAccept) srep->is_accept = acc;
          if (rec) rec->next_entry = ne;
          store_stats(J.stats[r], wst, nsteps);
        }
        __syncwarp();
        reinterpret_cast<int *>(J.rep + r)[lane] = sw[lane];
      }
    }
    if constexpr (MODE != 2) __syncthreads();
  }
}

}  // namespace gd

#include "gd_team.cuh"
#include "gd_spec.cuh"

namespace gd {

// Replica exchange between adjacent temperatures.  Sweep x pairs (t, t+1) for
// t = x mod 2, x mod 2 + 2, ... in every (protein conf p, ligand conf l)
// group; replica index n_tmp*n_lig*p + n_lig*t + l (src/frontend/util.C:380).
// Pair k of the sweep of job J:
__device__ void exchange_one(const DevJob &J, int x, int k)
{
  const int npair = (J.ntmp - (x & 1)) / 2;
  if (npair <= 0) return;
  const int ngroup = J.nprt * J.nlig;
  if (k >= ngroup * npair) return;
  const int g = k / npair, i = k % npair;
  const int p = g / J.nlig, l = g % J.nlig;
  const int t = (x & 1) + 2 * i;
  const int ga = J.ntmp * J.nlig * p + J.nlig * t + l;
  const int gb = ga + J.nlig;
  const int ra = ga - J.rid_base, rb = gb - J.rid_base;
  if (ra < 0 || rb >= J.nrep) return;
  ReplicaMC *A = J.rep + ra, *B = J.rep + rb;
  const Philox4 d = philox4x32_10((uint32_t)x, (uint32_t)g, 1u, (uint32_t)t, J.key0, J.key1);
  const double u = (double)u01(d.v[0]);
  const double ba = -(double)J.minus_beta[t], bb = -(double)J.minus_beta[t + 1];
  const double lr = (ba - bb) * ((double)A->energy[9] - (double)B->energy[9]);
  J.stats[ra].n_exch_try += 1;
  J.stats[rb].n_exch_try += 1;
  if (log(u) < lr) {
#pragma unroll
    for (int q = 0; q < 10; ++q) {
      const float tmp = A->energy[q];
      A->energy[q] = B->energy[q];
      B->energy[q] = tmp;
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const float tmp = A->movematrix[q];
      A->movematrix[q] = B->movematrix[q];
      B->movematrix[q] = tmp;
    }
    J.run_acc[ra] = 1;
    J.run_acc[rb] = 1;
    J.stats[ra].n_exch_acc += 1;
    J.stats[rb].n_exch_acc += 1;
  }
}

__global__ void exchange_kernel(const DevJob *jobp, int x)
{
  exchange_one(*jobp, x, blockIdx.x * blockDim.x + threadIdx.x);
}

// One sweep over every job of an ensemble.  xoff[parity][j] is the prefix sum
// of the pair counts (groups x pairs of that parity).  The sweep index is x, or
// with d_step the sweep that ends the chunk [*d_step, *d_step + chunk).
__global__ void exchange_all_kernel(const DevJob *jobs, const int *xoff, int njob, int x, const int *d_step,
                                    int spx, int chunk)
{
  if (d_step) x = (*d_step + chunk) / spx - 1;
  const int *off = xoff + (x & 1) * (njob + 1);
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= off[njob]) return;
  int lo = 0, hi = njob;  // off[lo] <= tid < off[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= tid) lo = mid;
    else hi = mid;
  }
  exchange_one(jobs[lo], x, tid - off[lo]);
}

// One sweep per job with the job's own sweep index (jobs admitted at
// different times are at different steps): blockIdx.y is the job.
__global__ void exchange_jobs_kernel(const DevJob *jobs)
{
  const DevJob &J = jobs[blockIdx.y];
  if (J.xsweep < 0) return;
  exchange_one(J, J.xsweep, blockIdx.x * blockDim.x + threadIdx.x);
}

__global__ void advance_step_kernel(int *d_step, int n) { *d_step += n; }
__global__ void set_step_kernel(int *d_step, int v) { *d_step = v; }

// ---------------------------------------------------------- launchers --
size_t kernel_smem_bytes(int P, int Pall, int lig_slots, int precision, const TileConfig &tc)
{
  return smem_layout(P, Pall, lig_slots, tc.warps_per_cta, precision == kFP64, tc.group, tc.split).total;
}

using McKernel = void (*)(KArgs);

// The kernel of a launch: the team form with several warps per replica, else
// the one-warp form of the tile shape.  FP64 has one shape, (1, 8).
template <int MODE, int PREC>
static McKernel pick_kernel(const TileConfig &tc)
{
  if (tc.group >= 8 && PREC != kFP64) return team_kernel<MODE, PREC, PREC != kFP64>;
  if (tc.group > 1) return team_kernel<MODE, PREC, false>;
  if constexpr (PREC == kFP64) return tc.kpl == 1 && tc.ab == 8 ? mc_kernel<MODE, PREC, 1, 8> : nullptr;
  else {
    // mode 2: the default shape, and (2, 8) with compensated sums for gd_noalloc.cu
    if constexpr (MODE != 2 || PREC == kFP32Kahan)
      if (tc.kpl == 2 && tc.ab == 8) return mc_kernel<MODE, PREC, 2, 8>;
    if constexpr (MODE != 2) {
      if (tc.kpl == 2 && tc.ab == 4) return mc_kernel<MODE, PREC, 2, 4>;
      if (tc.kpl == 4 && tc.ab == 4) return mc_kernel<MODE, PREC, 4, 4>;
    }
    if (tc.kpl == 4 && tc.ab == 8) return tc.wide ? mc_kernel<MODE, PREC, 4, 8, true> : mc_kernel<MODE, PREC, 4, 8>;
    return nullptr;
  }
}

static McKernel pick_kernel(int mode, int precision, const TileConfig &tc)
{
  if (mode == 0) {
    if (precision == kFP32) return pick_kernel<0, kFP32>(tc);
    if (precision == kFP32Kahan) return pick_kernel<0, kFP32Kahan>(tc);
    if (precision == kFP64) return pick_kernel<0, kFP64>(tc);
  } else if (mode == 2) {
    if (precision == kFP32) return pick_kernel<2, kFP32>(tc);
    if (precision == kFP32Kahan) return pick_kernel<2, kFP32Kahan>(tc);
    if (precision == kFP64) return pick_kernel<2, kFP64>(tc);
  } else {
    if (precision == kFP32) return pick_kernel<1, kFP32>(tc);
    if (precision == kFP32Kahan) return pick_kernel<1, kFP32Kahan>(tc);
    if (precision == kFP64) return pick_kernel<1, kFP64>(tc);
  }
  return nullptr;
}

// The kernel of a chunk on clusters (gd_spec.cuh); teams of 8 and 16 warps only.
static McKernel pick_spec(int precision)
{
  if (precision == kFP32) return spec_kernel<kFP32, true>;
  if (precision == kFP32Kahan) return spec_kernel<kFP32Kahan, true>;
  if (precision == kFP64) return spec_kernel<kFP64, false>;
  return nullptr;
}

// Lets kernel f be launched with `bytes` of dynamic shared memory in the current context.  The limit asked for only
// rises: a thread that needs less must not take it from under another's launch.  It is set at every launch, since it
// belongs to the context, and a process may have several or reset one.
static cudaError_t allow_smem(McKernel f, size_t bytes)
{
  static std::mutex mu;
  static std::map<McKernel, size_t> asked;
  std::lock_guard<std::mutex> lk(mu);
  size_t &most = asked[f];
  const cudaError_t s = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)std::max(bytes, most));
  if (s == cudaSuccess) most = std::max(bytes, most);
  return s;
}

struct SpecLaunch {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  cudaError_t prepare(McKernel k, const TileConfig &tc, int items, size_t smem, cudaStream_t st)
  {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = tc.cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(items * tc.cluster));
    cfg.blockDim = dim3((unsigned)(tc.warps_per_cta * 32));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = allow_smem(k, smem);
    if (e != cudaSuccess || tc.cluster <= 8) return e;
    return cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  }
};

// Occupancies of this process: they depend on the device, the kernel and the launch
// alone, whatever the context, and a small pose call looks up more of them (45 us) than its kernel
// takes.  Emptied when it has grown past any set of shapes in use.
static int known_occupancy(McKernel f, int cluster, const TileConfig &tc, size_t smem, int (*look)(McKernel, const TileConfig &, size_t))
{
  struct Key {
    McKernel f;
    size_t smem;
    int dev, warps, cluster;
    bool operator<(const Key &o) const
    {
      return std::tie(f, smem, dev, warps, cluster) < std::tie(o.f, o.smem, o.dev, o.warps, o.cluster);
    }
  };
  static std::mutex mu;
  static std::map<Key, int> known;
  Key k{f, smem, 0, tc.warps_per_cta, cluster};
  if (!f || cudaGetDevice(&k.dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lk(mu);
  const auto it = known.find(k);
  if (it != known.end()) return it->second;
  const int n = look(f, tc, smem);
  if (n > 0) {  // a failure may be of the moment
    if (known.size() >= 4096) known.clear();
    known[k] = n;
  }
  return n;
}

int cluster_occupancy(int precision, const TileConfig &tc, size_t smem)
{
  return known_occupancy(pick_spec(precision), tc.cluster, tc, smem, [](McKernel f, const TileConfig &t, size_t bytes) {
    SpecLaunch l;
    int n = 0;
    if (l.prepare(f, t, 1, bytes, nullptr) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, (const void *)f, &l.cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;
    }
    return n;
  });
}

cudaError_t launch_kernel(int mode, int precision, const TileConfig &tc, const KArgs &a, int grid, cudaStream_t st)
{
  const bool spec = mode == 0 && tc.cluster > 1 && a.nsteps > 1 && !(a.flags & kMcInitial);
  const McKernel k = spec ? pick_spec(precision) : pick_kernel(mode, precision, tc);
  if (!k) return cudaErrorInvalidValue;
  const size_t smem = kernel_smem_bytes(a.P, a.Pall, a.lig_slots, precision, tc);
  KArgs b = a;
  b.group = (uint8_t)tc.group;
  b.split = (uint8_t)tc.split;
  if (spec) {
    SpecLaunch l;
    const cudaError_t e = l.prepare(k, tc, a.n_items, smem, st);
    return e != cudaSuccess ? e : cudaLaunchKernelEx(&l.cfg, k, b);
  }
  const cudaError_t e = allow_smem(k, smem);
  if (e != cudaSuccess) return e;
  k<<<grid, tc.warps_per_cta * 32, smem, st>>>(b);
  return cudaGetLastError();
}

int kernel_occupancy(int mode, int precision, const TileConfig &tc, size_t smem)
{
  return known_occupancy(pick_kernel(mode, precision, tc), 1, tc, smem, [](McKernel f, const TileConfig &t, size_t bytes) {
    int nb = 0;
    if (allow_smem(f, bytes) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, f, t.warps_per_cta * 32, bytes) != cudaSuccess) return 0;
    return nb;
  });
}

cudaError_t launch_exchange_all(const DevJob *d_jobs, const int *d_xoff, int njob, int total, int x,
                                const int *d_step, int spx, int chunk, cudaStream_t st)
{
  if (total <= 0) return cudaSuccess;
  exchange_all_kernel<<<(total + 255) / 256, 256, 0, st>>>(d_jobs, d_xoff, njob, x, d_step, spx, chunk);
  return cudaGetLastError();
}

cudaError_t launch_exchange_jobs(const DevJob *d_jobs, int njob, int max_pairs, cudaStream_t st)
{
  if (njob <= 0 || max_pairs <= 0) return cudaSuccess;
  exchange_jobs_kernel<<<dim3((max_pairs + 127) / 128, njob), 128, 0, st>>>(d_jobs);
  return cudaGetLastError();
}

cudaError_t launch_set_step(int *d_step, int v, cudaStream_t st)
{
  set_step_kernel<<<1, 1, 0, st>>>(d_step, v);
  return cudaGetLastError();
}

cudaError_t launch_advance_step(int *d_step, int n, cudaStream_t st)
{
  advance_step_kernel<<<1, 1, 0, st>>>(d_step, n);
  return cudaGetLastError();
}

cudaError_t launch_exchange(const DevJob *d_job, int ngroup, int ntmp, int x, cudaStream_t st)
{
  const int npair = (ntmp - (x & 1)) / 2;
  if (npair <= 0 || ngroup <= 0) return cudaSuccess;
  const int n = ngroup * npair;
  exchange_kernel<<<(n + 255) / 256, 256, 0, st>>>(d_job, x);
  return cudaGetLastError();
}

}  // namespace gd

// Bounds-check record of the debug build: out4 = {1 if an index was out of
// range, its site (gd::CheckSite), the index, the array length}; reset != 0
// clears it.  The product build returns GD_E_STATE.
extern "C" int gd_check_report(int *out4, int reset)
{
  if (!out4) return gd::fail(GD_E_INVALID, "null argument");
#ifdef GD_CHECK
  GD_CUDA(cudaDeviceSynchronize());
  GD_CUDA(cudaMemcpyFromSymbol(out4, gd::g_check, 4 * sizeof(int)));
  if (reset) {
    const int z[4] = {0, 0, 0, 0};
    GD_CUDA(cudaMemcpyToSymbol(gd::g_check, z, sizeof z));
  }
  return GD_OK;
#else
  (void)reset;
  for (int i = 0; i < 4; ++i) out4[i] = 0;
  return gd::fail(GD_E_STATE, "not a bounds-checking build (libgdock_check.so is built with -DGD_CHECK)");
#endif
}

#ifdef GD_CHECK
namespace gd {
// The FP64 pair loop's functions: out[5 i] the reciprocal of x[i], its square root and half the reciprocal of that
// (x > 0), and the exponential of z[i] with and without the table's second part.
__global__ void math64_kernel(int n, const double *x, const double *z, double *out)
{
  __shared__ double tab[2 * kExpTab];
  for (int j = threadIdx.x; j < kExpTab; j += blockDim.x) exp_table_entry(tab, j);
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double *o = out + 5 * (size_t)i;
    o[0] = rcp64(x[i]);
    sqrt64(x[i], o[1], o[2]);
    o[3] = exp64<true>(z[i], tab);
    o[4] = exp64<false>(z[i], tab);
  }
}
}  // namespace gd
// The same for device arrays, in the bounds-checking build alone.
extern "C" int gd_check_math64(int n, const double *d_x, const double *d_z, double *d_out)
{
  if (n < 1 || !d_x || !d_z || !d_out) return gd::fail(GD_E_INVALID, "null argument");
  gd::math64_kernel<<<64, 256>>>(n, d_x, d_z, d_out);
  GD_CUDA(cudaDeviceSynchronize());
  return GD_OK;
}
#endif
