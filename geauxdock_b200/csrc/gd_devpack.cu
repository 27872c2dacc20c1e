// gd_devpack.cu -- packing a reference-layout Complex that is already in
// device memory into the kernels' structure-of-arrays layout, on the GPU.
//
// The same work as the host packer (gd_pack.cu: the semantics of the
// reference's OptimizeLigand / OptimizeProtein / OptimizePsp / OptimizeKde /
// OptimizeMcs / OptimizeEnepara, src/frontend/util_optimize_soa.C:37-540),
// with the same orders, so that both packings of one Complex are identical
// byte for byte:
//   - ligand atoms grouped by type, stable (util_optimize_soa.C:112-126), the
//     types with a hydrogen-bond parameter first;
//   - pocket points with the hydrophobic-contact flag first; in each part the
//     point types with a hydrogen-bond parameter first, each group sorted by
//     point type, stable; padded with inert points (type 30, far away);
//   - KDE points of ligand types sorted by type, stable, with per-type ranges
//     (util_optimize_soa.C:336-372; points of other types cannot match);
//   - MCS templates atom-major in grouped order, validity as energy_mcs_v1.cu;
//   - pocket-specific potential gathered per sorted class-2 point.
// Two callers: the allocation-free pose evaluation (destination: one static
// scratch array, gd_noalloc.cu) and Dock's refill of its resident state after
// CopyH2D put the next Complex on the GPU (destination: the arenas of the
// cached ensemble, gd_api.cu).  Invalid input sets the destination's error
// words; the kernels downstream check the flag and leave the job unread.
#include "gd_pack.h"

namespace gd {
namespace {

__device__ void dp_fail(const PackDst &D, int kind, int field, int value)
{
  if (atomicCAS(&D.err[1], 0, kind) == 0) {
    D.err[2] = field;
    D.err[3] = value;
  }
  atomicOr(&D.err[0], kErrPack);
}

// Sizes of the Complex, the same in every block; ok only where they are valid and
// those the destination holds.  Block 0 reports what is wrong.
struct DpSizes {
  int ok, nlig, nprt, ntmp, L, K, M, P;  // P: padded points per conformation
};

__device__ void dp_sizes(const Complex *cx, const PackDst &D, DpSizes &s)
{
  __shared__ int s_conf, s_point, s_max;  // first ligand conformation of another atom count, first bad point count
  const int tid = threadIdx.x;
  if (tid == 0) {
    s.nlig = cx->size.n_lig;
    s.nprt = cx->size.n_prt;
    s.ntmp = cx->size.n_tmp;
    s.K = cx->size.kde_npoint;
    s.M = cx->size.mcs_nrow;
    s.L = cx->lig[0].lig_natom;
    s_conf = s_point = 1 << 30;
    s_max = 0;
  }
  __syncthreads();
  if (tid < s.nlig && tid < GD_MAX_CONF_LIG && cx->lig[tid].lig_natom != s.L) atomicMin(&s_conf, tid);
  if (tid < s.nprt && tid < GD_MAX_CONF_PRT) {
    const int n = cx->prt[tid].prt_npoint;
    if (n < 1 || n > GD_MAXPRO) atomicMin(&s_point, tid);
    else atomicMax(&s_max, n);
  }
  __syncthreads();
  if (tid == 0) {
    int kind = 0, field = 0, value = 0;
    auto bad = [&](int k, int f, int v) {
      if (kind == 0) kind = k, field = f, value = v;
    };
    auto range = [&](int v, int lo, int hi, int f) {
      if (v < lo || v > hi) bad(v < lo ? kPackFailInput : kPackFailCapacity, f, v);
    };
    auto want = [&](int v, int expect, int f, int tell) {
      if (expect >= 0 && v != expect) bad(kPackFailShape, f, tell);
    };
    range(s.nlig, 1, GD_MAX_CONF_LIG, kFieldNLig);
    range(s.nprt, 1, GD_MAX_CONF_PRT, kFieldNPrt);
    range(s.L, 1, GD_MAXLIG, kFieldNatom);
    range(s.K, 0, GD_MAXKDE, kFieldKde);
    range(s.M, 1, GD_MAX_MCS_ROW, kFieldMcs);
    if (D.rep && (s.ntmp < 1 || s.ntmp > GD_MAX_TMP)) bad(kPackFailInput, kFieldNTmp, s.ntmp);
    if (kind == 0 && s_conf < s.nlig) bad(kPackFailInput, kFieldNatomConf, s_conf);
    if (kind == 0 && s_point < s.nprt) range(cx->prt[s_point].prt_npoint, 1, GD_MAXPRO, kFieldNpoint);
    s.P = ((s_max + kPointAlign - 1) / kPointAlign) * kPointAlign;
    want(s.P, D.Ppad > 0 ? D.Ppad : -1, kFieldNpoint, s_max);
    want(s.L, D.expect_L, kFieldNatom, s.L);
    want(s.nlig, D.expect_nlig, kFieldNLig, s.nlig);
    want(s.nprt, D.expect_nprt, kFieldNPrt, s.nprt);
    want(s.M, D.expect_M, kFieldMcs, s.M);
    if (D.rep) want(s.ntmp, D.expect_ntmp, kFieldNTmp, s.ntmp);
    if (D.rep && (D.rep_begin < 0 || D.rep_begin + D.nrep > cx->size.n_rep))
      bad(kPackFailShape, kFieldReplica, D.rep_begin + D.nrep);
    s.ok = kind == 0;
    if (kind && blockIdx.x == 0) dp_fail(D, kind, field, value);
  }
  __syncthreads();
}

// Bit pt of point[lt]'s union: the point types, and bit lt the ligand types, with
// a hydrogen-bond parameter (hdb0 > 0.1).
__device__ void dp_hdb_types(const Complex *cx, uint32_t &points, uint32_t &ligands)
{
  __shared__ uint32_t s_p, s_l;
  if (threadIdx.x == 0) s_p = s_l = 0u;
  __syncthreads();
  for (int q = threadIdx.x; q < kLigTypes * kPadType; q += blockDim.x) {
    const int lt = q / kPadType, pt = q % kPadType;
    if (cx->enepara.hdb0[lt][pt] > 0.1f) {
      atomicOr(&s_p, 1u << pt);
      atomicOr(&s_l, 1u << lt);
    }
  }
  __syncthreads();
  points = s_p;
  ligands = s_l;
}

// Ligand atoms grouped by type, the types with a hydrogen-bond parameter first,
// each part by type (stable): perm[k] = input index of grouped atom k; and each
// type's atoms [range & 0xffff, range >> 16).  An atom of an invalid type keeps
// its place in the order of the others (block 0 reports it).
__device__ void dp_ligand_order(const Complex *cx, int L, uint32_t hdb_ligands, int *perm, int *ltype, int *range)
{
  __shared__ int s_type[GD_MAXLIG];
  const int a = threadIdx.x;
  if (a < kLigTypes) range[a] = 0;
  if (a < L) {
    const int t = cx->lig[0].t2[a];
    s_type[a] = t >= 0 && t < kLigTypes ? t : 0;
  }
  __syncthreads();
  auto key = [&](int t) { return (((hdb_ligands >> t) & 1u) ? 0 : 32) + t; };
  int t = 0, r = 0, beg = 0, end = 0;
  if (a < L) {
    t = s_type[a];
    const int k = key(t);
    for (int b = 0; b < L; ++b) {
      const int kb = key(s_type[b]);
      r += kb < k || (kb == k && b < a);
      beg += kb < k;
      end += kb <= k;
    }
    perm[r] = a;
    ltype[r] = t;
    range[t] = beg | (end << 16);
  }
  __syncthreads();
}

// Block 0: validation of the ligand and the templates, force-field tables, ligand
// atom groups, centres, KDE slots, and the DevJob header (read only where the
// error flag stays clear).
__device__ void dp_setup(const Complex *cx, const PackDst &D, const DpSizes &s)
{
  __shared__ int s_kcnt[kLigTypes], s_kbeg[kLigTypes], s_slot[kLigTypes], s_nk, s_nslot;
  __shared__ int s_perm[GD_MAXLIG], s_ltype[GD_MAXLIG], s_range[kLigTypes];
  __shared__ unsigned char s_kt[GD_MAXKDE];  // KDE point types (255: none of the ligand's types)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int L = s.L, K = s.K, M = s.M, nlig = s.nlig, nprt = s.nprt;
  for (int a = tid; a < L; a += blockDim.x) {
    const int t = cx->lig[0].t2[a];
    if (t < 0 || t >= kLigTypes) dp_fail(D, kPackFailInput, kFieldLigType, a);
  }
  for (int m = warp; m < M; m += nwarps) {
    bool any = false;
    for (int a = lane; a < L; a += 32) any |= cx->mcs[m].x[a] != GD_MCS_INVALID_COORD;
    if (!__any_sync(0xffffffffu, any) && lane == 0) dp_fail(D, kPackFailInput, kFieldMcsRow, m);
  }
  uint32_t hp, hl;
  dp_hdb_types(cx, hp, hl);
  dp_ligand_order(cx, L, hl, s_perm, s_ltype, s_range);

  // force-field tables, as the host packer's build_params
  const EnePara &ep = cx->enepara;
  DevParams &par = *D.par;
  for (int q = tid; q < kLigTypes * kTabCols; q += blockDim.x) {
    const int lt = q / kTabCols, pt = q % kTabCols;
    if (pt < kPadType) {
      if (!(ep.p1a[lt][pt] > 0.f)) dp_fail(D, kPackFailInput, kFieldP1a, q);
      par.tab4[lt][pt] = tab4_entry(ep.p1a[lt][pt], ep.p2a[lt][pt], ep.pmf0[lt][pt], ep.pmf1[lt][pt]);
      const float h0 = ep.hdb0[lt][pt], h1 = ep.hdb1[lt][pt];
      const bool on = h0 > 0.1f;
      par.tab2[lt][pt] = on ? make_float2((float)((double)h1 * kHdbC), (float)(-(double)h0 * (double)h1 * kHdbC))
                            : make_float2(0.f, 0.f);
      D.ref4[q] = make_float4(ep.p1a[lt][pt], ep.p2a[lt][pt], on ? h0 : 0.f, on ? h1 : 0.f);
    } else {
      par.tab4[lt][pt] = tab4_padding();
      par.tab2[lt][pt] = make_float2(0.f, 0.f);
      D.ref4[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  for (int q = warp; q < kLigTypes; q += nwarps) {
    const uint32_t m = __ballot_sync(0xffffffffu, lane < kPadType && ep.hdb0[q][lane] > 0.1f);
    if (lane == 0) {
      par.hpl0[q] = ep.hpl0[q];
      par.hpl1[q] = ep.hpl1[q];
      par.hpl2[q] = ep.hpl2[q];
      par.hdbmask[q] = m;
    }
  }
  for (int q = tid; q < 12; q += blockDim.x) {
    par.a_para[q] = q < GD_MAXWEI ? ep.a_para[q] : 0.f;
    par.b_para[q] = q < GD_MAXWEI ? ep.b_para[q] : 0.f;
    par.w[q] = q < GD_MAXWEI ? ep.w[q] : 0.f;
  }
  if (tid == 0) {
    par.lj0 = ep.lj0;
    par.lj1 = ep.lj1;
    par.el0 = ep.el0;
    par.el1 = ep.el1;
    par.inv_el1 = 1.0f / ep.el1;
    par.a1 = ep.a1;
    par.b1 = ep.b1;
    par.kde2 = ep.kde2;
    par.kde3_inv = 1.0f / ep.kde3;
    par.lj01 = (float)((double)ep.lj0 * ep.lj1);
    par.ele_a = (float)((double)ep.a1 * ep.el1 * ep.el1);
    par.ele_b = (float)((double)ep.b1 * ep.el1 * ep.el1 * ep.el1);
    par.ele_d2max = (float)(1.0 / ((double)ep.el1 * ep.el1));
    par.hdb_cinv = (float)(1.0 / kHdbC);
    par.kde3 = ep.kde3;
    par.pad_ = 0.f;
  }
  for (int q = tid; q < 6; q += blockDim.x) par.move_scale[q] = cx->mcpara.move_scale[q];
  for (int a = tid; a < L; a += blockDim.x) D.lgrp[a] = make_int2(s_ltype[a], s_range[s_ltype[a]] >> 16);
  for (int q = tid; q < nlig * 3; q += blockDim.x) D.lcenter[q] = cx->lig[q / 3].center[q % 3];
  for (int q = tid; q < nprt * 3; q += blockDim.x) D.pcenter[q] = cx->prt[q / 3].pocket_center[q % 3];
  for (int q = tid; q < M; q += blockDim.x) D.tcc[q] = cx->mcs[q].tcc;

  // KDE points of ligand types, sorted by type (stable), and slots in the grouped
  // ligand's type order, one per KDE point of a type the ligand has: count, prefix, scatter
  for (int k = tid; k < K; k += blockDim.x) {
    const int t = cx->kde.t[k];
    s_kt[k] = t >= 0 && t < kLigTypes ? (unsigned char)t : (unsigned char)255;
  }
  __syncthreads();
  for (int t = warp; t < kLigTypes; t += nwarps) {
    int cnt = 0;
    for (int k0 = 0; k0 < K; k0 += 32) cnt += __popc(__ballot_sync(0xffffffffu, k0 + lane < K && s_kt[k0 + lane] == t));
    if (lane == 0) s_kcnt[t] = cnt;
  }
  __syncthreads();
  if (tid == 0) {
    int b = 0, o = 0;
    for (int t = 0; t < kLigTypes; ++t) {
      s_kbeg[t] = s_kcnt[t] ? b : 0;
      b += s_kcnt[t];
    }
    for (int a = 0; a < L; a = s_range[s_ltype[a]] >> 16) {
      s_slot[s_ltype[a]] = o;
      o += s_kcnt[s_ltype[a]];
    }
    s_nk = b;
    s_nslot = o;
    if (D.nkde_expect >= 0 && b != D.nkde_expect) dp_fail(D, kPackFailShape, kFieldKde, b);
  }
  __syncthreads();
  for (int t = warp; t < kLigTypes; t += nwarps) {
    int at = 0;
    const int range = s_range[t];
    const float inv = 1.0f / (float)s_kcnt[t];
    for (int k0 = 0; k0 < K; k0 += 32) {
      const int k = k0 + lane;
      const bool m = k < K && s_kt[k] == t;
      const unsigned b = __ballot_sync(0xffffffffu, m);
      const int rank = at + __popc(b & ((1u << lane) - 1u)), o = s_kbeg[t] + rank;
      if (m && o < D.kde_cap) {
        const float x = cx->kde.x[k], y = cx->kde.y[k], z = cx->kde.z[k];
        if (D.kde) D.kde[o] = make_float4(x, y, z, __int_as_float(t));
        const int q = s_slot[t] + rank;
        if (range && q < D.kde_cap) {
          D.kslot[2 * q] = make_int4(__float_as_int(x), __float_as_int(y), __float_as_int(z), __float_as_int(inv));
          D.kslot[2 * q + 1] = make_int4(range, s_kcnt[t], 0, 0);
        }
      }
      at += __popc(b);
    }
  }
  if (tid == 0 && s_nk == 0 && D.kde && D.kde_cap > 0) D.kde[0] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (tid < kLigTypes) {
    D.job->kbeg[tid] = s_kbeg[tid];
    D.job->kcnt[tid] = s_kcnt[tid];
    D.job->trange[tid] = s_range[tid];
  }
  if (tid == 0) {
    DevJob &J = *D.job;
    J.natom = L;
    J.nlig = nlig;
    J.lstride = (L + 3) & ~3;
    J.lig = D.lig;
    J.lgrp = D.lgrp;
    J.lcenter = D.lcenter;
    J.npoint_pad = s.P;
    J.nprt = nprt;
    J.pos = D.pos;
    J.aux = D.aux;
    J.ncdc = D.ncdc;
    J.pcenter = D.pcenter;
    J.psp = D.psp;
    J.pspmask = D.pspmask;
    J.pcell = D.pcell;
    J.pcell_cnt = D.pcell_cnt;
    J.pcell_stride = D.pcell_stride;
    J.pcell4 = D.pcell4;
    J.psp_table = &cx->psp.psp[0][0];
    J.nkde = s_nk;
    J.kde = D.kde;
    J.nkslot = min(s_nslot, D.kde_cap);
    J.kslot = D.kslot;
    J.nmcs = M;
    J.mcs = D.mcs;
    J.tcc = D.tcc;
    J.ntmp = D.rep ? s.ntmp : 0;
    J.minus_beta = D.minus_beta;
    J.par = D.par;
    J.ref4 = D.ref4;
    J.nrep = D.rep ? D.nrep : 0;
    J.rep = D.rep;
    J.run_acc = D.run_acc;
    J.stats = D.stats;
    J.rec = D.rec;
    J.key0 = D.key0;
    J.key1 = D.key1;
    J.rid_base = D.rep ? D.rep_begin : 0;
    J.nrep_total = D.rep ? D.nrep_total : 0;
    J.step0 = 0;
    J.nsteps = 0;
    J.xsweep = -1;
    J.pad_ = 0;
  }
}

// One block per protein conformation: points ordered as the host packer orders
// them (hydrophobic-contact points first, each part by hydrogen-bond group and
// point type, stable: 60 buckets counted and ranked with warp ballots), inert
// padding, the pocket-specific potential gathered with its non-zero type mask,
// and its non-zero cells for the ligand's types, by type then point.
__device__ void dp_pocket(const Complex *cx, const PackDst &D, const DpSizes &s, int i)
{
  constexpr int kBuckets = 2 * kPadType;
  __shared__ unsigned char s_key[GD_MAXPRO];
  __shared__ short s_src[GD_MAXPRO];       // input index of sorted point j
  __shared__ uint32_t s_mask[GD_MAXPRO];   // ligand types with a potential at sorted point j
  __shared__ int s_cnt[kBuckets], s_beg[kBuckets], s_ccnt[kLigTypes], s_cbeg[kLigTypes];
  __shared__ int s_perm[GD_MAXLIG], s_ltype[GD_MAXLIG], s_range[kLigTypes];
  const Protein &pr = cx->prt[i];
  const int np = pr.prt_npoint, Pp = s.P;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  uint32_t hp, hl;
  dp_hdb_types(cx, hp, hl);
  dp_ligand_order(cx, s.L, hl, s_perm, s_ltype, s_range);
  for (int k = tid; k < np; k += blockDim.x) {
    const int t = pr.t[k];
    int rank = kBuckets;  // an invalid type: left out
    if (t < 0 || t >= kPadType) {
      dp_fail(D, kPackFailInput, kFieldPrtType, k);
    } else {
      const uint32_t below = (1u << t) - 1u;
      rank = (pr.cdc[k] == 1 ? 0 : kPadType) +
             (((hp >> t) & 1u) ? __popc(hp & below) : __popc(hp) + t - __popc(hp & below));
    }
    s_key[k] = (unsigned char)rank;
  }
  for (int j = tid; j < Pp; j += blockDim.x) s_src[j] = -1;
  __syncthreads();
  for (int bk = warp; bk < kBuckets; bk += nwarps) {
    int cnt = 0;
    for (int k0 = 0; k0 < np; k0 += 32) cnt += __popc(__ballot_sync(0xffffffffu, k0 + lane < np && s_key[k0 + lane] == bk));
    if (lane == 0) s_cnt[bk] = cnt;
  }
  __syncthreads();
  if (tid == 0) {
    int b = 0, nc = 0;
    for (int q = 0; q < kBuckets; ++q) {
      s_beg[q] = b;
      b += s_cnt[q];
      if (q < kPadType) nc += s_cnt[q];
    }
    D.ncdc[i] = nc;
  }
  __syncthreads();
  for (int bk = warp; bk < kBuckets; bk += nwarps) {
    int at = s_beg[bk];
    if (s_cnt[bk] == 0) continue;
    for (int k0 = 0; k0 < np; k0 += 32) {
      const int k = k0 + lane;
      const bool m = k < np && s_key[k] == bk;
      const unsigned b = __ballot_sync(0xffffffffu, m);
      if (m) s_src[at + __popc(b & ((1u << lane) - 1u))] = (short)k;
      at += __popc(b);
    }
  }
  __syncthreads();
  float4 *pos = D.pos + (size_t)i * Pp;
  float2 *aux = D.aux + (size_t)i * Pp;
  for (int j = tid; j < Pp; j += blockDim.x) {
    const int k = s_src[j];
    uint32_t mask = 0u;
    if (k >= 0) {
      pos[j] = make_float4(pr.x[k], pr.y[k], pr.z[k], pr.ele[k]);
      aux[j] = make_float2(pr.cdc[k] == 1 ? pr.hpp[k] : 0.f, __int_as_float(pr.t[k]));
      int col = -1;
      if (pr.c[k] == 2) {
        col = pr.seq3r[k];
        if (col < 0 || col >= GD_MAXPRO) {
          dp_fail(D, kPackFailInput, kFieldSeq3r, k);
          col = -1;
        }
      }
      if (col >= 0)
#pragma unroll
        for (int lt = 0; lt < kLigTypes; ++lt) mask |= (cx->psp.psp[lt][col] != 0.f ? 1u : 0u) << lt;
    } else {
      pos[j] = make_float4(1.0e4f + (float)j, 1.0e4f, 1.0e4f, 0.f);
      aux[j] = make_float2(0.f, __int_as_float(kPadType));
    }
    s_mask[j] = mask;
    if (D.pspmask) D.pspmask[(size_t)i * Pp + j] = mask;
  }
  __syncthreads();
  if (D.psp) {
    float *psp = D.psp + (size_t)i * kLigTypes * Pp;
    for (int lt = warp; lt < kLigTypes; lt += nwarps)
      for (int j = lane; j < Pp; j += 32)
        psp[(size_t)lt * Pp + j] = ((s_mask[j] >> lt) & 1u) ? cx->psp.psp[lt][pr.seq3r[s_src[j]]] : 0.f;
  }
  // cells of the ligand's types: the atoms of type t are s_range[t]
  if (warp < kLigTypes) {
    int nc = 0;
    if (s_range[warp])
      for (int j0 = 0; j0 < Pp; j0 += 32)
        nc += __popc(__ballot_sync(0xffffffffu, (s_mask[j0 + lane] >> warp) & 1u));
    if (lane == 0) s_ccnt[warp] = nc;
  }
  __syncthreads();
  if (tid == 0) {
    int c = 0;
    for (int t = 0; t < kLigTypes; ++t) {
      s_cbeg[t] = c;
      c += s_ccnt[t];
    }
    D.pcell_cnt[i] = min(c, D.pcell_stride);
    if (c > D.pcell_stride) dp_fail(D, kPackFailCapacity, kFieldPcell, c);
  }
  __syncthreads();
  if (warp < kLigTypes && s_ccnt[warp] > 0) {
    const int t = warp;
    int at = s_cbeg[t];
    for (int j0 = 0; j0 < Pp; j0 += 32) {
      const int j = j0 + lane;
      const bool m = (s_mask[j] >> t) & 1u;
      const unsigned b = __ballot_sync(0xffffffffu, m);
      const int o = at + __popc(b & ((1u << lane) - 1u));
      if (m && o < D.pcell_stride) {
        const int k = s_src[j], col = pr.seq3r[k];
        if (D.pcell) {
          int4 *cell = D.pcell + ((size_t)i * D.pcell_stride + o) * 2;
          cell[0] = make_int4(__float_as_int(pr.x[k]), __float_as_int(pr.y[k]), __float_as_int(pr.z[k]),
                              __float_as_int(cx->psp.psp[t][col]));
          cell[1] = make_int4(s_range[t], __float_as_int(-cx->enepara.pmf0[t][pr.t[k]]), t, j);
        } else {
          D.pcell4[(size_t)i * D.pcell_stride + o] = pack_cell4(j, t, col);
        }
      }
      at += __popc(b);
    }
  }
}

// The other blocks: ligand conformations in grouped atom order, MCS templates
// atom-major; with a replica destination also the replica range, accept flags,
// statistics and the temperature ladder.
__device__ void dp_ligand(const Complex *cx, const PackDst &D, const DpSizes &s, int block, int nblock)
{
  __shared__ int s_perm[GD_MAXLIG], s_ltype[GD_MAXLIG], s_range[kLigTypes];
  const int L = s.L, M = s.M, nlig = s.nlig, nprt = s.nprt, ntmp = s.ntmp;
  const int ls = (L + 3) & ~3;
  uint32_t hp, hl;
  dp_hdb_types(cx, hp, hl);
  dp_ligand_order(cx, L, hl, s_perm, s_ltype, s_range);
  const int stride = nblock * blockDim.x;
  const int g = block * blockDim.x + threadIdx.x;
  for (int q = g; q < nlig * ls; q += stride) {
    const int i = q / ls, a = q % ls;
    if (a < L) {
      const int k = s_perm[a];
      const Ligand &lg = cx->lig[i];
      D.lig[q] = make_float4(lg.x2[k], lg.y2[k], lg.z2[k], cx->lig[0].c2[k]);
    } else {
      D.lig[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  for (int q = g; q < L * M; q += stride) {
    const int a = q / M, m = q % M;
    const int k = s_perm[a];
    const float x = cx->mcs[m].x[k];
    D.mcs[q] = make_float4(x, cx->mcs[m].y[k], cx->mcs[m].z[k], x != GD_MCS_INVALID_COORD ? 1.f : 0.f);
  }
  if (!D.rep) return;
  for (int t = g; t < ntmp; t += stride) D.minus_beta[t] = cx->temp[t].minus_beta;
  for (int r = g; r < D.nrep; r += stride) {
    ReplicaMC R = cx->replica[D.rep_begin + r];
    if (R.idx_lig < 0 || R.idx_lig >= nlig || R.idx_prt < 0 || R.idx_prt >= nprt || R.idx_tmp < 0 ||
        R.idx_tmp >= ntmp) {
      dp_fail(D, kPackFailInput, kFieldReplica, D.rep_begin + r);
      R.idx_lig = R.idx_prt = R.idx_tmp = 0;  // in range, whatever reads it before the flag is seen
    }
    D.rep[r] = R;
    int *words = reinterpret_cast<int *>(D.rep + r);
    for (int i = kReplicaUsed / 4; i < (int)(sizeof(ReplicaMC) / 4); ++i) words[i] = 0;
    D.run_acc[r] = R.is_accept;
    RepStats S;
    S.e_sum = S.e_sum2 = S.best_e = 0.0;
    S.n_steps = S.n_accept = S.n_exch_try = S.n_exch_acc = 0;
    for (int i = 0; i < 6; ++i) S.best_mm[i] = 0.f;
    S.best_step = -1;
    S.pad_ = 0;
    D.stats[r] = S;
  }
}

// The whole packing in one launch: no block needs another's output (each works
// out the sizes, the hydrogen-bond types and the ligand's order for itself, 720
// parameters and up to 64 atoms), so nothing waits between them.  What bounds it
// is the latency of each block's few dependent passes over global memory; as
// three launches whose orders and checks ran on one thread it took 110 + 70 + 30
// us for 40 atoms x 1500 points x 11 conformations, now 33 us
// (as a refill of Dock's state, with replicas and the dense potential, 260 -> 44 us).
constexpr int kPackLigBlocks = 16;
__global__ void __launch_bounds__(1024) dp_pack_kernel(const Complex *__restrict__ cx, PackDst D)
{
  __shared__ DpSizes s;
  dp_sizes(cx, D, s);
  if (!s.ok) return;
  const int b = blockIdx.x;
  if (b == 0) dp_setup(cx, D, s);
  else if (b <= GD_MAX_CONF_PRT) {
    if (b <= s.nprt) dp_pocket(cx, D, s, b - 1);
  } else dp_ligand(cx, D, s, b - 1 - GD_MAX_CONF_PRT, kPackLigBlocks);
}

}  // namespace

cudaError_t device_pack(const Complex *d_cx, const PackDst &D, cudaStream_t st)
{
  (void)cudaGetLastError();  // a failure an earlier call already reported is not this launch's
  dp_pack_kernel<<<1 + GD_MAX_CONF_PRT + kPackLigBlocks, 1024, 0, st>>>(d_cx, D);
  return cudaGetLastError();
}

const char *pack_field_name(int f)
{
  switch (f) {
    case kFieldNLig: return "size.n_lig (ligand conformations)";
    case kFieldNPrt: return "size.n_prt (protein conformations)";
    case kFieldNatom: return "lig[0].lig_natom (ligand atoms)";
    case kFieldNatomConf: return "a ligand conformation's lig_natom (differs from conformation 0)";
    case kFieldNpoint: return "prt[i].prt_npoint (protein points)";
    case kFieldKde: return "size.kde_npoint (KDE points)";
    case kFieldMcs: return "size.mcs_nrow (MCS rows)";
    case kFieldLigType: return "a ligand atom type (index given)";
    case kFieldPrtType: return "a protein point type (index given)";
    case kFieldSeq3r: return "a class-2 point's seq3r (index given)";
    case kFieldMcsRow: return "an MCS row without any coordinate (row given)";
    case kFieldP1a: return "enepara.p1a <= 0 (index lt * 32 + pt given; the pair kernel needs p1a > 0)";
    case kFieldNTmp: return "size.n_tmp (temperatures)";
    case kFieldReplica: return "a replica's conformation or temperature index (replica given)";
    case kFieldPcell: return "non-zero pocket-specific cells of a conformation";
    default: return "unknown field";
  }
}

}  // namespace gd
