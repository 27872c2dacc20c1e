// gd_team.cuh -- the batched kernel's other form: one replica (or pose) on a
// team of G warps of a CTA, for launches whose replicas alone would leave most
// of the GPU idle.
//
// A step is a chain of dependent work that one warp takes ~36 us for (24 atoms x
// 600 points) whatever else the GPU does; the only way to shorten it is to
// spread the step.  Each warp of the team keeps its own copy of the replica's
// pose, draws the same random numbers (16 steps at a time, one lane per step
// and counter word) and rotates its own copy of the ligand, so that a step
// costs two barriers: after the units of the energy -- pair-loop rows, contact
// blocks, chunks of the KDE and pocket-specific walks, the MCS templates --
// dealt out to the warps in turn, and after the nine terms, each combined from
// its units by one warp.
//
// The units and the order they are combined in are the one-warp kernel's
// (split order V = 1) or those of a replica split over V = 2, 4 or 8 warps
// (option replica_warps: rows, KDE and pocket cells, contact rows and templates
// dealt out to V shares, summed share by share), whatever the team's size: the
// results depend on V alone and the host chooses G by what fits one wave.
//
// A step of 24 atoms x 600 points takes 7.1 us on 16 warps (one warp 36 us, the
// former split over 8 warps 17 us), of 34 x 344 over 51 replicas 7.5 us (42 us).
// It is bound by one SM's special-function and issue rate for the rows (~9,300
// of 13,900 cycles, ten half rows on four schedulers) and by the two barriers'
// serial parts (combining ~2,300, rotation 1,000, finishing 500).  FP32 <-> FP64
// conversions are kept out of the step's common path: every warp finishing the
// terms through doubles cost 2,500 cycles.  In the split order of 8 the 49 sums of
// shares go up to four to a warp through one butterfly (one after the other 1,000
// cycles a step more), and the warp with the templates sits out the first turns of
// the other tasks (3,000 less where the templates end last).
#pragma once

#include "gd_energy.cuh"

namespace gd {

// Barrier of the G warps of one team (named barrier 1 + index of the team).
__device__ __forceinline__ void team_sync(int team, int G)
{
  asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(G * 32) : "memory");
}

// What the energy of a pose reads besides the job: the work item's shared data.
struct ItemData {
  const DevParams *par;
  const float4 *pos;
  const float2 *aux;
  const int2 *lgrp;
  const float4 *apt, *aph;
  const int4 *ahd;
};

// A team's shared memory.
template <int PREC>
struct TeamArea {
  using T = RealOf<PREC>;
  ReplicaMC *rep;
  WarpStats *stats;
  T *part;     // [9][8] the terms: the scaled sum of each share, or (V = 1, and the distance) the term as it is and normalised
  T *mcs;      // MCS sums of the shares, and in [8] the squared distance of the centres
  T *rows;     // pass 1 per lane: [rows][4][32] vdw, ele, pmf, hdb, or [rows][2][7][32] the components (HalfRow)
  T *contact;  // [V][kMaxAtoms] hydrophobic-contact sums
  T *walk[2];  // KDE, pocket-specific: [chunks][32][2] terms, then [V][32] sums
  __device__ TeamArea(unsigned char *base, const SmemLayout &sl, int nrows, int row_reals, int V, int chunks)
  {
    rep = reinterpret_cast<ReplicaMC *>(base);
    stats = reinterpret_cast<WarpStats *>(base + sizeof(ReplicaMC));
    part = reinterpret_cast<T *>(base + sizeof(ReplicaMC) + sizeof(WarpStats));
    mcs = part + 72;
    rows = reinterpret_cast<T *>(base + sl.parts);
    contact = rows + row_reals * nrows;
    walk[0] = contact + V * kMaxAtoms;
    walk[1] = walk[0] + 64 * chunks + 32 * V;
  }
};

// (double)x by its bits where x is a normal number: all warps of a team convert
// the same two energies every step, and conversion instructions to and from
// FP64 issue at ~2 lanes per clock and SM.
__device__ __forceinline__ double to_double(float x)
{
  const uint32_t u = __float_as_uint(x), ex = (u >> 23) & 255u;
  if (ex == 0u || ex == 255u) return (double)x;
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
}

// Term k of the KDE (which = 0) or pocket-specific walk.
template <int PREC, bool C4>
__device__ __forceinline__ WalkTerm<RealOf<PREC>> team_walk_term(const DevJob &J, const DevParams *par,
                                                              const LigOf<PREC> *lig, int which, int iprt, int k)
{
  if (which == 0) return kde_slot<PREC>(J.kslot, J.nkde, J.natom, kde_exponent<PREC>(par), lig, k);
  if constexpr (C4) return psp_cell4<PREC>(J, iprt, lig, k);
  else return psp_cell<PREC>(J.pcell + (size_t)iprt * J.pcell_stride * 2, J.pcell_stride, J.natom, lig, k);
}

__device__ __forceinline__ int walk_length(const DevJob &J, int which, int iprt)
{
  return which == 0 ? J.nkslot : J.pcell_cnt[iprt];
}

// Task `task` of `ntask` of a walk: the terms of its chunks or, without chunks,
// the lanes' sums of the share that is the task.
template <int PREC, bool C4>
__device__ __forceinline__ void team_walk(const DevJob &J, const DevParams *par, const TeamArea<PREC> &A,
                                          const LigOf<PREC> *lig, int which, int iprt, int task, int ntask, int chunks)
{
  using T = RealOf<PREC>;
  const int lane = lane_id(), n = walk_length(J, which, iprt);
  T *w = A.walk[which];
  T acc = 0;
#pragma unroll 1
  for (int c = task; 32 * c < n && (chunks == 0 || c < chunks); c += ntask) {
    WalkTerm<T> t{0, 0};
    if (32 * c + lane < n) t = team_walk_term<PREC, C4>(J, par, lig, which, iprt, 32 * c + lane);
    if (chunks) {
      w[64 * c + lane] = t.x;
      w[64 * c + 32 + lane] = t.w;
    } else if (32 * c + lane < n) {
      acc = fma_(t.x, t.w, acc);
    }
  }
  if (chunks == 0) w[32 * task + lane] = acc;
}

template <int PREC, int KPL, bool DEEP>
__device__ __forceinline__ float4 team_row_sums(const LigPair *lig, int npairs, int row, int P, const ItemData &D)
{
  return pass1_row<KPL, DEEP>(lig, npairs, row, P, D.pos, D.aux, D.apt, D.aph, D.ahd, PairConst::load(D.par));
}
__device__ __forceinline__ void team_half_sums(const LigPair *lig, int npairs, int c, int row, int P, const ItemData &D,
                                            float *o)
{
  const HalfRow h = pass1_half(lig, npairs, c, row, P, D.pos, D.aux, D.apt, D.aph, D.ahd, PairConst::load(D.par));
  o[0] = h.vdw;
  o[32] = h.pmf;
  o[64] = h.hdb;
#pragma unroll
  for (int j = 0; j < 4; ++j) o[96 + 32 * j] = h.ele[j];
}

__device__ __forceinline__ void kahan_add_any(float &s, float &c, float x) { kahan_add(s, c, x); }
__device__ __forceinline__ void kahan_add_any(double &s, float &, double x) { s = add_(s, x); }

// Task t of combining a team's units: share v of term i (the contact, 5, has one).
__device__ __forceinline__ void team_task(int t, int V, int &i, int &v)
{
  const int q = t >> (31 - __clz(V));  // V is a power of two
  i = t == 6 * V ? 5 : q == 5 ? 6 : q;
  v = t == 6 * V ? 0 : t - q * V;
}

// A finished term: as it is, and normalised.
template <int PREC>
__device__ __forceinline__ void team_term(RealOf<PREC> *part, int i, RealOf<PREC> raw, const DevParams *par, int L)
{
  part[8 * i] = raw;
  part[8 * i + 1] = norm_term(i, raw, par, L);
}

// A level of two butterflies at once: a lane whose bit o is clear goes on with the
// first pair (s0, c0), the others with the second, in (s0, c0); with the same
// pair twice, a level of warp_sum_pair (FP64: warp_sum).
__device__ __forceinline__ void sum_merge(float &s0, float &c0, float s1, float c1, int o)
{
  const bool hi = (lane_id() & o) != 0;
  const float s = hi ? s1 : s0, c = hi ? c1 : c0;
  const float so = __shfl_xor_sync(0xffffffffu, hi ? s0 : s1, o), co = __shfl_xor_sync(0xffffffffu, hi ? c0 : c1, o);
  const float t = add_(s, so), bp = sub_(t, s);
  c0 = add_(add_(c, co), add_(sub_(s, sub_(t, bp)), sub_(so, bp)));
  s0 = t;
}
__device__ __forceinline__ void sum_merge(double &s0, float &, double s1, float, int o)
{
  const bool hi = (lane_id() & o) != 0;
  const double s = hi ? s1 : s0;
  s0 = add_(s, __shfl_xor_sync(0xffffffffu, hi ? s0 : s1, o));
}

// Energy of ligand conformation ilig at the pose in pm (lane k < 6 holds
// movematrix[k]) in protein conformation iprt by the team's warps: on return
// lane i < 9 of every warp holds term i, normalised in e and before that in raw,
// and every lane the total (SOLO: of the first warp alone; the finishing of 16
// warps costs them each other's issue slots).  What the next call writes before
// its first barrier nobody but the first warp reads after this call's second.
template <int PREC, bool WIDE, bool C4, bool SOLO = false>
__device__ __forceinline__ RealOf<PREC> team_energy(const DevJob &J, const ItemData &D, const TeamArea<PREC> &A,
                                                    LigOf<PREC> *lig, int team, int sub, int G, int V, int chunks,
                                                    int ilig, int iprt, float pm, RealOf<PREC> &e, RealOf<PREC> &raw)
{
  using T = RealOf<PREC>;
  const int lane = lane_id(), L = J.natom, P = J.npoint_pad;
  rotate_ligand<PREC>(J, ilig, pm, lig);

  // rows dealt out first; the shorter tasks go to the warps a last incomplete round of rows leaves over
  constexpr bool kHalves = WIDE && PREC != kFP64;
  const bool halves = kHalves && V == 1;
  const int row = team_row(V), nr = P / row, nrt = halves ? 2 * nr : nr;
  for (int t = sub; t < nrt; t += G) {
    if constexpr (PREC == kFP64) {
      T *o = A.rows + 128 * t + lane;
      double h[4];
      pass1_row64(lig, L, D.lgrp, D.par, reinterpret_cast<const double2 *>(D.apt), D.aph,
                  reinterpret_cast<const double *>(D.ahd), t * row, P, D.pos, D.aux, h);
#pragma unroll
      for (int k = 0; k < 4; ++k) o[32 * k] = h[k];
    } else {
      const int np = (L + 1) >> 1;
      if (halves) {
        team_half_sums(lig, np, t & 1, (t >> 1) * row, P, D, A.rows + 224 * t + lane);
      } else {
        T *o = A.rows + 128 * t + lane;
        float4 h;
        if (kHalves || V > 1) h = team_row_sums<PREC, 2, WIDE>(lig, np, t * row, P, D);
        else h = team_row_sums<PREC, 4, false>(lig, np, t * row, P, D);
        o[0] = h.x;
        o[32] = h.y;
        o[64] = h.z;
        o[96] = h.w;
      }
    }
  }
  const int nb = (L + kContactBlock - 1) / kContactBlock;
  const int crows = contact_rows(J, iprt), nv = min(V, max(1, crows / kHalfPoints));  // shares with a contact row
  const int nw = chunks ? 4 : V;  // tasks of a walk
  // task 0 takes as long as four or five of the others, so its warp sits out the first four turns of those
  const int t1 = nb * nv, t2 = t1 + 2 * nw, busy = nrt % G, W = G - busy, x = sub - busy;
  for (int turn = 0, next = 1; x >= 0 && next <= t2; ++turn) {
    const int first = turn < 4 ? 1 : 0, t = turn == 0 && x == 0 ? 0 : x < first ? t2 + 1 : next + x - first;
    next += W - first;
    if (t > t2) continue;
    if (t == 0) {
      // the longest of them
      const T m = mcs_sums<PREC>(J, lig, V, A.mcs), dst = centre_dist2<T>(J, ilig, iprt, pm);
      if (lane == 0) {
        if (V == 1) A.mcs[0] = m;
        A.mcs[8] = dst;
      }
    } else if (t <= t1) {
      const int v = (t - 1) / nb, a0 = kContactBlock * (t - 1 - v * nb), a = a0 + (lane >> 2);
      const T S = contact_block<PREC, kContactBlock>(lig, L, a0, kHalfPoints * v, kHalfPoints * V, crows, D.pos, D.aux, P);
      if ((lane & 3) == 0 && a < L) A.contact[v * kMaxAtoms + a] = S;
    } else {
      const int which = t - t1 > nw;
      team_walk<PREC, C4>(J, D.par, A, lig, which, iprt, t - t1 - 1 - which * nw, nw, chunks);
    }
  }
  team_sync(team, G);

  // terms 0..6 from their units, dealt out to the warps: per share of V the lanes' sums (the rows' with the
  // compensation c) and a butterfly, up to four of a warp's in one
  for (int t0 = sub; t0 < 6 * V + 1; t0 += 4 * G) {
    T s4[4] = {0, 0, 0, 0};
    float c4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int q = 0; q < 4 && t0 + q * G < 6 * V + 1; ++q) {
      int i, v;
      team_task(t0 + q * G, V, i, v);
      T s = 0;
      float c = 0.f;
      if (i < 5 && i != 3) {
        // the rows' sums; the two components of a row joined as pass1_row does
        const T *u = A.rows + (halves ? 32 * (i == 1 ? 3 : i >> 1) : 32 * (i == 4 ? 3 : i)) + lane;
#pragma unroll 2
        for (int r = v; r < nr; r += V) {
          T h;
          if (!halves) {
            h = u[128 * r];
          } else if (i != 1) {
            h = add_(u[448 * r], u[448 * r + 224]);
          } else {
            h = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
              h = fma_((T)D.pos[r * row + 32 * j + lane].w, add_(u[448 * r + 32 * j], u[448 * r + 224 + 32 * j]), h);
          }
          // a plain sum is the compensated one without c
          kahan_add_any(s, c, h);
        }
      } else if (i != 5) {
        const T *w = A.walk[i == 3] + lane;
        if (chunks == 0) {
          s = w[32 * v];
        } else {
          const int n = walk_length(J, i == 3, iprt);
#pragma unroll 2
          for (int k = 0; k < chunks && 32 * k < n; ++k)
            if (32 * k + lane < n) s = fma_(w[64 * k], w[64 * k + 32], s);
#pragma unroll 1
          for (int k = 32 * chunks + lane; k < n; k += 32) {  // past the chunks kept
            const WalkTerm<T> x = team_walk_term<PREC, C4>(J, D.par, lig, i == 3, iprt, k);
            s = fma_(x.x, x.w, s);
          }
        }
      } else {
        // a lane's atoms and their order: those of the one-warp kernel's blocks, or one lane per atom
        const bool blocks = V == 1;
        if (!blocks || (lane & 3) == 0)
#pragma unroll 1
          for (int a = blocks ? lane >> 2 : lane; a < L; a += blocks ? kContactBlock : 32) {
            T S = A.contact[a];
            for (int k = 1; k < nv; ++k) S = add_(S, A.contact[k * kMaxAtoms + a]);
            s = add_(s, contact_restraint(D.par, D.lgrp, a, L, S));
          }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        s4[k] = q == k ? s : s4[k];
        c4[k] = q == k ? c : c4[k];
      }
    }
    sum_merge(s4[0], c4[0], s4[1], c4[1], 16);
    sum_merge(s4[2], c4[2], s4[3], c4[3], 16);
    sum_merge(s4[0], c4[0], s4[2], c4[2], 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) sum_merge(s4[0], c4[0], s4[0], c4[0], o);
    const int t = t0 + (2 * ((lane >> 3) & 1) + (lane >> 4)) * G;
    if ((lane & 7) == 0 && t < 6 * V + 1) {
      int i, v;
      team_task(t, V, i, v);
      T x = s4[0];
      if (PREC == kFP32Kahan && i < 3) x = add_(x, (T)c4[0]);  // the dense terms are compensated
      x = scaled_sum<PREC>(i, x, D.par);
      if (V > 1) A.part[8 * i + v] = x;
      else team_term<PREC>(A.part, i, i == 4 ? raw_term<PREC>(4, x, J.nmcs) : x, D.par, L);
    }
  }
  if (sub == G - 1) {
    if (lane < V) {
      if (V > 1) A.part[8 * 7 + lane] = A.mcs[lane];
      else team_term<PREC>(A.part, 7, raw_term<PREC>(7, A.mcs[0], J.nmcs), D.par, L);
    }
    if (lane == 8) team_term<PREC>(A.part, 8, raw_term<PREC>(8, A.mcs[8], J.nmcs), D.par, L);
  }
  team_sync(team, G);
  if (SOLO && sub > 0) return 0;

  // every warp: lane i has term i, finished where it was summed, or (V > 1) adds its shares in order (dense terms
  // compensated) and finishes it; the weighted total in term order
  const int i = min(lane, 8);
  const T *p = A.part + 8 * i;
  raw = p[0];
  e = p[1];
  if (V > 1 && i != 8) {
    T x = raw;
    float c = 0.f;
#pragma unroll
    for (int v = 1; v < 8; ++v)
      if (v < V && i != 5) kahan_add_any(x, c, p[v]);
    if (PREC == kFP32Kahan && i < 3) x = add_(x, (T)c);
    raw = i == 4 || i == 7 ? raw_term<PREC>(i, x, J.nmcs) : x;
    e = norm_term(i, raw, D.par, L);
  }
  T tot = 0;
#pragma unroll
  for (int k = 0; k < 9; ++k) tot = fma_((T)D.par->w[k], __shfl_sync(0xffffffffu, e, k), tot);
  return tot;
}

// Random numbers of steps [s, s + kDrawSteps) of replica r by one warp, the counters
// of the one-warp kernel: lane 2 q + w has word w of step s + q.  Row q of draw:
// the six moves and two unused words; logu: the logarithm of the acceptance draw.
__device__ __forceinline__ void draw_steps(const DevJob &J, int r, int s, float *draw, double *logu)
{
  const int lane = lane_id();
  const Philox4 d = philox4x32_10((uint32_t)(s + (lane >> 1)), (uint32_t)(J.rid_base + r), 0u, (uint32_t)(lane & 1),
                                  J.key0, J.key1);
  float *o = draw + 8 * (lane >> 1) + 4 * (lane & 1);
  o[0] = u01(d.v[0]);
  o[1] = u01(d.v[1]);
  o[2] = u01(d.v[2]);
  o[3] = u01(d.v[3]);
  if (lane & 1) logu[lane >> 1] = log((double)u01(d.v[2]));
}

// Metropolis test in FP64, kernel_cuda_l1_montecarlo.cu:485-507.
__device__ __forceinline__ int team_accept(double logu, float etot, float ecur, double mbeta)
{
  return logu < (to_double(etot) - to_double(ecur)) * mbeta;
}

// A replica's state, statistics and Record during a chunk, kept by one warp of its
// team (state and statistics in shared memory).
struct TeamRecord {
  Record *rec;
  int acc, ne;  // accepted in the step before; Record entries

  __device__ __forceinline__ void begin(const KArgs &A, const DevJob &J, int r, ReplicaMC *srep, WarpStats *wst)
  {
    const int lane = lane_id();
    reinterpret_cast<int *>(srep)[lane] = reinterpret_cast<const int *>(J.rep + r)[lane];
    if (lane == 0) load_stats(wst, J.stats[r]);
    rec = (J.rec && (A.flags & kMcRecord)) ? J.rec + r : nullptr;
    acc = J.run_acc[r];
    ne = 0;
    if (J.rec && (A.flags & kMcResetRecord)) {
      if (lane == 0) J.rec[r].next_entry = 0;
    } else if (rec) {
      ne = rec->next_entry;
    }
    __syncwarp();
  }
  // Before step s: a state that was accepted is recorded, kernel_cuda_l1_montecarlo.cu:290-297.
  __device__ __forceinline__ void before(ReplicaMC *srep, int s)
  {
    if (!acc) return;
    const int lane = lane_id();
    if (lane == 0) srep->step = s;
    __syncwarp();
    if (rec && ne < GD_STEPS_PER_DUMP)
      reinterpret_cast<int *>(&rec->replica[ne])[lane] = reinterpret_cast<const int *>(srep)[lane];
    ++ne;
  }
  // After step s: lane k < 9 has term k in et, lane k < 6 word k of the pose in pm.
  __device__ __forceinline__ void after(ReplicaMC *srep, WarpStats *wst, int s, int accept, float et, float etot, float pm)
  {
    const int lane = lane_id();
    if (accept) {
      if (lane < 9) srep->energy[lane] = et;
      if (lane == 9) srep->energy[9] = etot;
      if (lane < 6) srep->movematrix[lane] = pm;
    }
    __syncwarp();
    if (lane == 0) step_stats(wst, accept, (double)srep->energy[9], s, srep->movematrix);
    acc = accept;
  }
  __device__ __forceinline__ void end(const KArgs &A, const DevJob &J, int r, ReplicaMC *srep, const WarpStats *wst,
                                      int nsteps)
  {
    const int lane = lane_id();
    if (lane == 0) {
      J.run_acc[r] = acc;
      if (A.flags & kMcStoreAccept) srep->is_accept = acc;
      if (rec) rec->next_entry = ne;
      store_stats(J.stats[r], wst, nsteps);
    }
    __syncwarp();
    reinterpret_cast<int *>(J.rep + r)[lane] = reinterpret_cast<const int *>(srep)[lane];
  }
};

// WIDE: teams of 8 and 16 warps, one CTA per SM: 128 registers, deep pair loops.
template <int MODE, int PREC, bool WIDE>
__global__ void __maxnreg__(PREC == kFP64 || WIDE ? 128 : 80) team_kernel(KArgs A)
{
  using T = RealOf<PREC>;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int s_item;
  const int G = A.group, V = A.split, chunks = V > 1 ? 0 : team_chunks(G);
  const SmemLayout sl = smem_layout(A.P, A.Pall, A.lig_slots, blockDim.x / 32, PREC == kFP64, G, V);
  const int warp = threadIdx.x >> 5, lane = lane_id();
  const int team = warp / G, sub = warp - team * G;
  // a Complex the device packer refused (gd_devpack.cu) leaves its job unread
  if (*(volatile int *)A.err & kErrPack) return;
  if (threadIdx.x == 0) mbar_init(&bar, 1);
  __syncthreads();
  uint32_t phase = 0;
  int prev_job = -1, prev_prt = -1;
  unsigned char *wbase = smem + sl.warp0 + (size_t)warp * sl.warp_bytes;
  LigOf<PREC> *lig = reinterpret_cast<LigOf<PREC> *>(wbase);
  // this warp's random numbers of kDrawSteps steps: six moves (and two unused words), log of the acceptance draw
  float *draw = reinterpret_cast<float *>(wbase + sl.lig_bytes);
  double *logu = reinterpret_cast<double *>(draw + 8 * kDrawSteps);

  for (int turn = 0;; ++turn) {
    const int it = next_item<MODE>(A, turn, &s_item);
    if (it >= A.n_items) break;
    const WorkItem wi = work_item<MODE>(A, it, (blockDim.x >> 5) / G);
    const DevJob &J = A.jobs[wi.job];
    if (!load_item<PREC>(A, J, wi, smem, sl, &bar, phase, prev_job, prev_prt)) return;
    ItemData D;
    D.par = reinterpret_cast<const DevParams *>(smem + sl.params);
    D.pos = A.P > 0 ? reinterpret_cast<const float4 *>(smem + sl.pos) : J.pos + (size_t)wi.prt * J.npoint_pad;
    D.aux = A.P > 0 ? reinterpret_cast<const float2 *>(smem + sl.aux) : J.aux + (size_t)wi.prt * J.npoint_pad;
    D.lgrp = reinterpret_cast<const int2 *>(smem + sl.lgrp);
    D.apt = reinterpret_cast<const float4 *>(smem + sl.apt);
    D.aph = reinterpret_cast<const float4 *>(smem + sl.aph);
    D.ahd = reinterpret_cast<const int4 *>(smem + sl.ahd);
    const TeamArea<PREC> T_(smem + sl.team0 + (size_t)team * sl.team_bytes, sl, A.Pall / team_row(V), team_row_reals(G, V, PREC == kFP64), V, chunks);

    if (team < wi.count) {
      const int r = wi.rep0 + team;  // job-local index
      if constexpr (MODE >= 1) {
        const int ilig = A.conf[2 * (size_t)r], iprt = A.conf[2 * (size_t)r + 1];
        if constexpr (MODE == 2) {
          if (bad_pose(A, J, r, ilig, iprt, sub == 0)) continue;  // the team alike; no CTA barrier follows
          D.pos = J.pos + (size_t)iprt * J.npoint_pad;
          D.aux = J.aux + (size_t)iprt * J.npoint_pad;
        }
        const float pm = lane < 6 ? A.mm[6 * (size_t)r + lane] : 0.0f;
        T et, raw;
        const T tot = team_energy<PREC, WIDE, MODE == 2>(J, D, T_, lig, team, sub, G, V, chunks, ilig, iprt, pm, et, raw);
        if (sub == 0) {
          const double e = (double)(lane < 9 ? et : tot);
          if (lane < 10) {
            A.out[10 * (size_t)r + lane] = (float)e;
            if (A.out64) A.out64[10 * (size_t)r + lane] = e;
          }
          if (A.raw && lane < 9) A.raw[9 * (size_t)r + lane] = (float)raw;
        }
      } else {
        // ---- Monte Carlo chunk for replica r; the team's first warp keeps its state
        const bool lead = sub == 0;
        const ReplicaMC *grep = J.rep + GD_AT(r, J.nrep, kSiteRep);
        float cur = lane < 6 ? grep->movematrix[lane] : 0.0f;  // every warp's copy of the pose and its total
        float ecur = grep->energy[9];
        const int ilig = grep->idx_lig, iprt = grep->idx_prt;
        const double mbeta = (double)J.minus_beta[GD_AT(grep->idx_tmp, J.ntmp, kSiteTmp)];
        TeamRecord R;
        if (lead) R.begin(A, J, r, T_.rep, T_.stats);
        const bool initial = (A.flags & kMcInitial) != 0;
        const int s0 = (A.d_step ? *A.d_step + A.s_begin : A.s_begin) + J.step0;
        const int nsteps = J.nsteps > 0 ? min(J.nsteps, A.nsteps) : A.nsteps;
        for (int k = 0; k < nsteps; ++k) {
          const int s = s0 + k, ks = k & (kDrawSteps - 1);
          if (ks == 0 && !initial) {
            __syncwarp();
            draw_steps(J, r, s, draw, logu);
            __syncwarp();
          }
          const float pm = lane < 6 ? __fmaf_rn(D.par->move_scale[lane], initial ? 0.0f : draw[8 * ks + lane], cur) : 0.0f;
          if (lead) R.before(T_.rep, s);
          T et, raw;
          const float etot =
              (float)team_energy<PREC, WIDE, MODE == 2>(J, D, T_, lig, team, sub, G, V, chunks, ilig, iprt, pm, et, raw);
          int accept = 1;
          if (!initial) accept = team_accept(logu[ks], etot, ecur, mbeta);
          if (accept) {
            ecur = etot;
            cur = pm;
          }
          if (lead) R.after(T_.rep, T_.stats, s, accept, (float)et, etot, pm);
        }
        if (lead) R.end(A, J, r, T_.rep, T_.stats, nsteps);
      }
    }
    if constexpr (MODE != 2) __syncthreads();
  }
}

}  // namespace gd
