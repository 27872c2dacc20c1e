// gd_spec.cuh -- a Monte Carlo chunk of a replica on several SMs, for launches
// that have fewer replicas than the GPU has SMs.
//
// A step cannot start before the step before it is decided, and one SM cannot
// make a step much shorter (gd_team.cuh).  But the proposals are known ahead:
// the random numbers are counters, and each step leaves the replica either where
// it was or at its proposal.  So the energies of the steps that may follow are
// evaluated at the same time, one node of the tree of decisions per CTA of
// a thread-block cluster, a team of warps each.  A round: every node's
// pose is built from the current one along its path, its energy evaluated as any
// other, the ten energies written to every CTA of the cluster (distributed shared
// memory, a transaction barrier in each), and then every warp makes the Metropolis
// tests of all nodes, one per lane, and follows their path from the root.  That
// makes exactly the decisions, states and Records that one step after the other
// makes.
//
// Which nodes: the most probable ones at the replica's rate of acceptance
// so far (spec_trees).  A round of 16 nodes is 4.8 steps at a rate of 0.26.
//
// A round of 24 atoms x 600 points takes 8.5 us, a step of a lone team 7.1: the
// energy as there, and 500 cycles for the pose, 700 for the nodes' energies to
// arrive and 900 for the tests.  A cluster barrier in place of the transaction
// barrier takes 2,200, the tests one after the other along the path 2,600, and all
// warps finishing the terms 1,200 more.  So a step is 1.8 us (one warp: 36 us).
//
// The wait for a round's energies is bounded as the staging waits are, by option
// wait_limit, but by no less than kNodeWaitNs: it spans other CTAs' work (a CTA without
// a node waits a whole energy).  A CTA that gives up leaves the rounds; the others
// miss it in the next one.  They then tell each other how many rounds each has sent,
// and each waits until all that was sent to it has arrived before it returns.
#pragma once

namespace gd {

constexpr int kSpecNodes = kMaxCluster;
constexpr int kSpecRates = 10;   // rates of acceptance 0.05, 0.15, ...
constexpr int kSpecRing = 64;    // steps whose random numbers are kept: a round and the next reach 31 steps ahead
constexpr int kSpecRoot = 255;
constexpr uint64_t kNodeWaitNs = 10000000ull;  // ten times the energy of 128 atoms x 20,000 points in FP64

// Nodes in the order of their probability, so that the first n are the best n
// and a node follows those on its path.
struct SpecNode {
  uint16_t path;      // bit j: the step j after the current one is accepted
  uint8_t depth;
  uint8_t base;       // the last node on the path that is accepted (kSpecRoot: none)
  uint16_t yes, no;   // the nodes on the path that are accepted, rejected
};
struct SpecTrees {
  SpecNode node[kSpecRates][kSpecNodes];
};
constexpr SpecTrees spec_trees()
{
  SpecTrees T{};
  for (int b = 0; b < kSpecRates; ++b) {
    const double rate = 0.05 + 0.1 * b;
    // candidates: the children of the nodes taken
    double prob[kSpecNodes + 1] = {1.0};
    SpecNode cand[kSpecNodes + 1] = {SpecNode{0, 0, kSpecRoot, 0, 0}};
    for (int k = 0; k < kSpecNodes; ++k) {
      int best = 0;
      for (int i = 1; i <= k; ++i)
        if (prob[i] > prob[best]) best = i;
      const SpecNode n = cand[best];
      const double p = prob[best];
      T.node[b][k] = n;
      prob[best] = p * (1.0 - rate);
      cand[best] = SpecNode{n.path, (uint8_t)(n.depth + 1), n.base, n.yes, (uint16_t)(n.no | (1 << k))};
      prob[k + 1] = p * rate;
      cand[k + 1] = SpecNode{(uint16_t)(n.path | (1 << n.depth)), (uint8_t)(n.depth + 1), (uint8_t)k,
                             (uint16_t)(n.yes | (1 << k)), n.no};
    }
  }
  return T;
}
static __device__ const SpecTrees kSpecTrees = spec_trees();

__device__ __forceinline__ int cluster_ctas()
{
  int n;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
  return n;
}
__device__ __forceinline__ int cluster_rank()
{
  int n;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(n));
  return n;
}
// All threads of the cluster; what was written before, also to other CTAs' shared memory, is seen after.
__device__ __forceinline__ void cluster_sync()
{
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// The address in CTA `rank`'s shared memory of this CTA's variable at p.
__device__ __forceinline__ uint32_t cluster_map(const void *p, int rank)
{
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_store(uint32_t a, int v)
{
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// The same, counted as 4 bytes on the barrier `bar` of that CTA.
__device__ __forceinline__ void cluster_store_tx(uint32_t a, float v, uint32_t bar)
{
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];" ::"r"(a),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}

// After some CTA of the cluster gave up (one thread): lets the energies still under way to this CTA arrive.  full: the
// rounds' barriers, of which this CTA has armed those of the rounds before `mine`; sent[c]: rounds that CTA c has sent
// (negative where it gave up).
// The others differ from `mine` by one at most: whoever sent a round had received all of the one before.
__device__ void spec_drain(uint64_t *full, int mine, bool complete, const int *sent, int ctas, uint32_t extra)
{
  int missing = 0, ahead = 0;
  for (int c = 0; c < ctas; ++c) {
    missing += abs(sent[c]) < mine;
    ahead += abs(sent[c]) > mine;
  }
  if (!complete) {
    const int last = mine - 1;
    if (missing || extra) mbar_complete_tx(&full[last & 1], 40u * missing + extra);
    (void)mbar_wait(&full[last & 1], (last >> 1) & 1, kWaitLimitNs);
  }
  if (ahead) {
    mbar_expect_tx(&full[mine & 1], 40u * ahead);
    (void)mbar_wait(&full[mine & 1], (mine >> 1) & 1, kWaitLimitNs);
  }
}

// One replica (a work item of one) per cluster; the CTA of rank c has node c.
template <int PREC, bool WIDE>
__global__ void __maxnreg__(128) spec_kernel(KArgs A)
{
  using T = RealOf<PREC>;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar, full[2];
  __shared__ SpecNode s_tree[kSpecRates][kSpecNodes];
  __shared__ double s_logu[kSpecRing];
  __shared__ float s_draw[8 * kSpecRing];
  __shared__ float s_node[2][kSpecNodes][12];  // a round's nodes: nine terms and the total; two rounds in turn
  __shared__ int s_fail, s_sent[kSpecNodes];
  const int G = A.group, V = A.split, chunks = V > 1 ? 0 : team_chunks(G);
  const int sub = threadIdx.x >> 5, lane = lane_id();
  const int ctas = cluster_ctas(), mine = cluster_rank();
  const SmemLayout sl = smem_layout(A.P, A.Pall, A.lig_slots, G, PREC == kFP64, G, V);
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    s_fail = 0;
  }
  __syncthreads();
  const WorkItem wi = A.items[blockIdx.x / ctas];
  const DevJob &J = A.jobs[wi.job];
  uint32_t phase = 0;
  int prev_job = -1, prev_prt = -1;
  // a Complex the device packer refused (gd_devpack.cu) leaves its job unread
  const int refused = __syncthreads_or(*(volatile int *)A.err & kErrPack);
  const bool fail = refused || !load_item<PREC>(A, J, wi, smem, sl, &bar, phase, prev_job, prev_prt);
  // the cluster's CTAs go on or return together: none writes to the shared memory of one that has returned
  cluster_sync();
  if (fail && threadIdx.x < ctas) cluster_store(cluster_map(&s_fail, threadIdx.x), 1);
  cluster_sync();
  if (s_fail) return;

  ItemData D;
  D.par = reinterpret_cast<const DevParams *>(smem + sl.params);
  D.pos = A.P > 0 ? reinterpret_cast<const float4 *>(smem + sl.pos) : J.pos + (size_t)wi.prt * J.npoint_pad;
  D.aux = A.P > 0 ? reinterpret_cast<const float2 *>(smem + sl.aux) : J.aux + (size_t)wi.prt * J.npoint_pad;
  D.lgrp = reinterpret_cast<const int2 *>(smem + sl.lgrp);
  D.apt = reinterpret_cast<const float4 *>(smem + sl.apt);
  D.aph = reinterpret_cast<const float4 *>(smem + sl.aph);
  D.ahd = reinterpret_cast<const int4 *>(smem + sl.ahd);
  const TeamArea<PREC> area(smem + sl.team0, sl, A.Pall / team_row(V),
                            team_row_reals(G, V, PREC == kFP64), V, chunks);
  LigOf<PREC> *lig = reinterpret_cast<LigOf<PREC> *>(smem + sl.warp0 + (size_t)sub * sl.warp_bytes);

  const int r = wi.rep0;
  const ReplicaMC *grep = J.rep + GD_AT(r, J.nrep, kSiteRep);
  float cur = lane < 6 ? grep->movematrix[lane] : 0.0f;  // every warp's copy of the pose and its total
  float ecur = grep->energy[9];
  const int ilig = grep->idx_lig, iprt = grep->idx_prt;
  const double mbeta = (double)J.minus_beta[GD_AT(grep->idx_tmp, J.ntmp, kSiteTmp)];
  const float scale = lane < 6 ? D.par->move_scale[lane] : 0.0f;
  const int s0 = (A.d_step ? *A.d_step + A.s_begin : A.s_begin) + J.step0;
  const int nsteps = J.nsteps > 0 ? min(J.nsteps, A.nsteps) : A.nsteps;
  // accepted and all steps that the rate is taken from: at most 64 earlier ones, and a prior of one in four
  const long long before = J.stats[r].n_steps;
  const float w = fminf((float)before, 64.f);
  float nacc = 1.f + (before > 0 ? w * ((float)J.stats[r].n_accept / (float)before) : 0.f), ntry = 4.f + w;
  // the replica's state is kept by a warp that the rows rarely reach, the random numbers drawn by another
  for (int i = threadIdx.x; i < kSpecRates * kSpecNodes; i += blockDim.x) (&s_tree[0][0])[i] = (&kSpecTrees.node[0][0])[i];
  const bool lead = mine == 0 && sub == G - 1, fill = sub == G - 2;
  TeamRecord R;
  if (lead) R.begin(A, J, r, area.rep, area.stats);
  int blocks = 0;
  if (fill)
    for (; blocks < 2; ++blocks)
      draw_steps(J, r, s0 + kDrawSteps * blocks, s_draw + 8 * kDrawSteps * blocks, s_logu + kDrawSteps * blocks);
  __syncthreads();

  const uint64_t limit = A.wait_limit ? max(wait_limit_ns(A.wait_limit), kNodeWaitNs) : kWaitLimitNs;
  const uint32_t extra = (A.flags & kMcStallNodes) && mine == ctas - 1 ? 16u : 0u;  // test hook
  bool alive = true;
  int round = 0;
  for (int k = 0; k < nsteps; ++round) {
    const SpecNode *tree = s_tree[max(0, min(kSpecRates - 1, (int)(kSpecRates * nacc / ntry)))];
    float (*nodes)[12] = s_node[round & 1];
    uint64_t *bar2 = &full[round & 1];
    if (threadIdx.x == 0) mbar_expect_tx(bar2, 40u * ctas + extra);
    if (fill)
      // the next round starts at step k + 16 at most and reaches 15 further
      for (; kDrawSteps * blocks <= k + 31; ++blocks) {
        const int o = kDrawSteps * blocks & (kSpecRing - 1);
        draw_steps(J, r, s0 + kDrawSteps * blocks, s_draw + 8 * o, s_logu + o);
      }
    const SpecNode me = tree[mine];
    float v = 0.0f;
    if (k + me.depth < nsteps) {
      float pm = cur;
      for (int path = me.path | 1 << me.depth; path; path &= path - 1)
        if (lane < 6) pm = __fmaf_rn(scale, s_draw[8 * ((k + __ffs(path) - 1) & (kSpecRing - 1)) + lane], pm);
      T et, raw;
      const T tot = team_energy<PREC, WIDE, false, true>(J, D, area, lig, 0, sub, G, V, chunks, ilig, iprt, pm, et, raw);
      v = lane < 9 ? (float)et : (float)tot;
    } else {
      // nothing to evaluate; as after an energy, the team has read the round before
      team_sync(0, G);
    }
    if (sub == 0 && lane < 10)
      for (int c = 0; c < ctas; ++c) cluster_store_tx(cluster_map(&nodes[mine][lane], c), v, cluster_map(bar2, c));
    // one decision for the whole CTA: a warp that gave up and one that did not must not go separate ways
    alive = __syncthreads_and(mbar_wait(bar2, (round >> 1) & 1, limit) ? 1 : 0) != 0;
    if (!alive) break;

    // lane n: the test of node n against the energy that its path leaves
    const SpecNode at = tree[lane & (kSpecNodes - 1)];
    const bool valid = lane < ctas && k + at.depth < nsteps;
    int accept = 0;
    if (valid)
      accept = team_accept(s_logu[(k + at.depth) & (kSpecRing - 1)], nodes[lane][9],
                           at.base == kSpecRoot ? ecur : nodes[at.base][9], mbeta);
    const uint32_t yes = __ballot_sync(0xffffffffu, accept);
    const uint32_t walk = __ballot_sync(0xffffffffu, valid && (yes & at.yes) == at.yes && (yes & at.no) == 0);
    const uint32_t took = yes & walk;
    const int count = __popc(walk);
    if (lead) {
      float pm0 = cur;
      uint32_t left = walk;
      for (int j = 0; j < count; ++j, left &= left - 1) {
        const int node = __ffs(left) - 1, s = k + j, ok = (took >> node) & 1;
        const float pm = lane < 6 ? __fmaf_rn(scale, s_draw[8 * (s & (kSpecRing - 1)) + lane], pm0) : 0.0f;
        R.before(area.rep, s0 + s);
        __syncwarp();
        R.after(area.rep, area.stats, s0 + s, ok, nodes[node][min(lane, 9)], nodes[node][9], pm);
        __syncwarp();
        if (ok) pm0 = pm;
      }
    }
    if (took) {
      const int node = 31 - __clz(took);
      ecur = nodes[node][9];
      for (int path = tree[node].path | 1 << tree[node].depth; path; path &= path - 1)
        if (lane < 6) cur = __fmaf_rn(scale, s_draw[8 * ((k + __ffs(path) - 1) & (kSpecRing - 1)) + lane], cur);
      nacc += (float)__popc(took);
    }
    ntry += (float)count;
    k += count;
  }
  if (lead && alive) R.end(A, J, r, area.rep, area.stats, nsteps);
  if (!alive && threadIdx.x == 0) atomicOr(A.err, kErrTimeout);
  // no CTA returns while another may still write to its shared memory
  const int sent = alive ? round : round + 1;
  if (threadIdx.x < ctas) cluster_store(cluster_map(&s_sent[mine], threadIdx.x), alive ? sent : -sent);
  cluster_sync();
  bool all = true;
  for (int c = 0; c < ctas; ++c) all &= s_sent[c] >= 0;
  if (all || threadIdx.x > 0) return;
  spec_drain(full, sent, alive, s_sent, ctas, extra);
}

}  // namespace gd
