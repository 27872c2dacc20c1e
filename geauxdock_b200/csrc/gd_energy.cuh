// gd_energy.cuh -- the parts of one pose's energy, shared by the kernels that
// give a pose one warp (gd_mc.cu) and a team of warps (gd_team.cuh).
//
// A pose's energy has the same bits in both.  The sums are cut into units whose
// arithmetic does not depend on who evaluates them -- 128-point rows of the pair
// loop, 8-atom blocks of the hydrophobic contact, 32-point chunks of the KDE and
// of the pocket-specific walk -- and the units are combined in the one-warp
// kernel's order (or both times in that of a split, where one is asked for).  Every multiply-add below is written out (__fmaf_rn and the
// like), so that the compiler's own contraction cannot differ between the two
// places a function is inlined.
#pragma once

#include <type_traits>

#include "gd_device.cuh"
#include "gd_internal.h"

namespace gd {

constexpr int kRowPoints = 128;   // points of a row of the one-warp pair loop (4 per lane)
constexpr int kHalfPoints = 64;   // points of a row of the split order and of the hydrophobic contact
constexpr int kContactBlock = 8;  // atoms of a hydrophobic-contact block

__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_(double a, double b) { return __dsub_rn(a, b); }

// Squared length, the operations of the pair loop in its order; and in the order of the KDE and MCS sums.
template <typename T>
__device__ __forceinline__ T dist2(T dx, T dy, T dz)
{
  return fma_(dx, dx, fma_(dy, dy, mul_(dz, dz)));
}
template <typename T>
__device__ __forceinline__ T dist2_xyz(T dx, T dy, T dz)
{
  return fma_(dz, dz, fma_(dx, dx, mul_(dy, dy)));
}

// The rotated ligand of one pose in shared memory: atom pairs in FP32, atoms in FP64.
template <int PREC>
using LigOf = typename std::conditional<PREC == kFP64, V4<double>, LigPair>::type;
template <int PREC>
using RealOf = typename std::conditional<PREC == kFP64, double, float>::type;

// Rotation + translation, kernel_cuda_l1_montecarlo.cu:336-380, by one warp;
// lane k < 6 holds movematrix[k] in pm.  The three angles' sines and cosines
// are evaluated by three lanes at once.
template <int PREC>
__device__ __forceinline__ void rotate_ligand(const DevJob &J, int ilig, float pm, LigOf<PREC> *lig)
{
  using T = RealOf<PREC>;
  const int lane = lane_id();
  const float ang = (lane >= 3 && lane < 6) ? pm : 0.0f;
  T s, c;
  if constexpr (PREC == kFP64) sincos((double)ang, &s, &c);
  else sincosf(ang, &s, &c);
  constexpr unsigned kAll = 0xffffffffu;
  const T s1 = __shfl_sync(kAll, s, 3), c1 = __shfl_sync(kAll, c, 3);
  const T s2 = __shfl_sync(kAll, s, 4), c2 = __shfl_sync(kAll, c, 4);
  const T s3 = __shfl_sync(kAll, s, 5), c3 = __shfl_sync(kAll, c, 5);
  const T c1c3 = mul_(c1, c3), c3s1 = mul_(c3, s1);
  const T r00 = mul_(c1, c2), r01 = fma_(mul_(c1, s2), s3, -c3s1), r02 = fma_(s1, s3, mul_(c1c3, s2));
  const T r10 = mul_(c2, s1), r11 = fma_(mul_(s1, s2), s3, c1c3), r12 = fma_(c3s1, s2, -mul_(c1, s3));
  const T r20 = -s2, r21 = mul_(c2, s3), r22 = mul_(c2, c3);
  const float *lc = J.lcenter + 3 * GD_AT(ilig, J.nlig, kSiteLigConf);
  const T tx = add_((T)__shfl_sync(kAll, pm, 0), (T)lc[0]), ty = add_((T)__shfl_sync(kAll, pm, 1), (T)lc[1]),
          tz = add_((T)__shfl_sync(kAll, pm, 2), (T)lc[2]);
  const int L = J.natom;
  const float4 *lsrc = J.lig + (size_t)ilig * J.lstride;
  for (int a = lane; a < L; a += 32) {
    const float4 v = lsrc[a];
    const T x = (T)v.x, y = (T)v.y, z = (T)v.z;
    const T ox = add_(fma_(r02, z, fma_(r00, x, mul_(r01, y))), tx);
    const T oy = add_(fma_(r12, z, fma_(r10, x, mul_(r11, y))), ty);
    const T oz = add_(fma_(r22, z, fma_(r21, y, mul_(r20, x))), tz);
    if constexpr (PREC == kFP64) {
      lig[a] = V4<double>{ox, oy, oz, (double)v.w};
    } else {
      float *f = reinterpret_cast<float *>(lig + (a >> 1)) + (a & 1);
      f[0] = ox;
      f[2] = oy;
      f[4] = oz;
      f[6] = v.w;
    }
  }
  if constexpr (PREC != kFP64) {
    // the dummy half of an odd atom count: far from every point (padding
    // points sit near +1e4), no charge; its table entries make every term 0
    if ((L & 1) && lane == 0) {
      float *f = reinterpret_cast<float *>(lig + (L >> 1)) + 1;
      f[0] = -1.0e4f;
      f[2] = -1.0e4f;
      f[4] = -1.0e4f;
      f[6] = 0.0f;
    }
  }
  __syncwarp();
}

// Scalar force-field constants of the pair terms, read once per pose.
struct PairConst {
  float lj0, lj01, el0, inv_el1, ea, eb, ed2;
  __device__ static PairConst load(const DevParams *p)
  {
    PairConst c;
    c.lj0 = p->lj0; c.lj01 = p->lj01; c.el0 = p->el0; c.inv_el1 = p->inv_el1;
    c.ea = p->ele_a; c.eb = p->ele_b; c.ed2 = p->ele_d2max;
    return c;
  }
};

// The same in FP64, and the exponential's table.
struct PairConst64 {
  double lj0, lj01, el0, inv_el1, ed2, ea, eb;
  const double *tab;
};

// -------------------------------------------- pair loop, FP32 (pass 1) --
// Protein-ligand pair terms but the hydrophobic contact, energy_prt_v1.cu:56-139.
//
// Running sums of one point row: component k of each float2 belongs to atom
// 2i + k of the pair being visited; the electrostatic term q_a q_p g(d) is
// summed per point as q_p * sum_a q_a g(d).
template <int KPL>
struct PairAccP {
  float2 vdw, pmf, hdb;
  float2 ele[KPL];
};

// Per work item, shared-memory tables of the atom-pair pair loop, built from
// the per-type tables (read from global memory): for pair i (atoms a = 2i,
// b = 2i + 1) and point type pt, e = i * kTabCols + pt,
//   apt[2e]     = (1/p1a, -p2a/p1a) of a and b interleaved: (a.x, b.x, a.y, b.y)
//   apt[2e + 1] = (-pmf0, pmf1) interleaved
//   aph[e]      = (hdb1 c, -hdb0 hdb1 c) interleaved
//   ahd[i]      = (point types with hydrogen-bond parameters for a or b,
//                  bit set of the types of a and b, type of a, type of b or 31).
// The dummy half of an odd atom count gets the padding column and no types:
// every term of it is exactly 0.
__device__ void build_pair_tables(int L, const DevParams *par, const int2 *lg, float4 *apt, float4 *aph, int4 *ahd)
{
  const int npairs = (L + 1) >> 1;
  for (int e = threadIdx.x; e < npairs * kTabCols; e += blockDim.x) {
    const int i = e / kTabCols, pt = e % kTabCols;
    const int a = 2 * i, b = a + 1;
    const int lta = GD_AT(lg[GD_AT(a, L, kSiteLgrp)].x, kLigTypes, kSiteTab), ltb = b < L ? lg[b].x : -1;
    const float4 ta = par->tab4[lta][pt];
    const float4 tb = ltb >= 0 ? par->tab4[ltb][pt] : tab4_padding();
    apt[2 * e] = make_float4(ta.x, tb.x, ta.y, tb.y);
    apt[2 * e + 1] = make_float4(ta.z, tb.z, ta.w, tb.w);
    const float2 ha = par->tab2[lta][pt], hb = ltb >= 0 ? par->tab2[ltb][pt] : make_float2(0.f, 0.f);
    aph[e] = make_float4(ha.x, hb.x, ha.y, hb.y);
    if (pt == 0) {
      const uint32_t hm = par->hdbmask[lta] | (ltb >= 0 ? par->hdbmask[ltb] : 0u);
      const uint32_t tb_bits = (1u << lta) | (ltb >= 0 ? 1u << ltb : 0u);
      ahd[i] = make_int4((int)hm, (int)tb_bits, lta, ltb >= 0 ? ltb : 31);
    }
  }
}

// Pair terms of ligand atom pair i against the lane's KPL points, two atoms per
// packed f32x2 instruction (__ffma2_rn / __fadd2_rn / __fmul2_rn, sm_100); the
// special functions stay per component.  FP32 uses rearranged forms of the
// reference's formulas:
//   LJ = (1 - (p2a/p1a) d^3) / (lj0 + lj0 lj1 d^2 + d^9 / p1a)   (divided through by p1),
//   g  = el0 + d^2 (a1 el1^2 + b1 el1^3 d) for el1 d < 1, else r/el1 with r = 1/d,
//   hdb1 exp(-((d - hdb0) hdb1)^2 / 2) = (hdb1 c) 2^-(d hdb1 c - hdb0 hdb1 c)^2 / c.
// HDB: evaluate the hydrogen-bond term (some point of the row has a parameter
// for one of the two atoms); the pocket-specific term is walked over its
// non-zero cells after the loop.  npx/npy/npz hold the lane's negated point
// coordinates twice (x_atom - x_point is x_atom + (-x_point), exactly); the
// charges are read from shared memory where they are used, which keeps the
// loop within its registers.
template <int KPL, bool HDB, bool DEEP>
__device__ __forceinline__ void pair_atom_pair(const LigPair *__restrict__ lig, int i GD_CHECK_ARG(int npairs), const float2 &lx,
                                               const float2 &ly, const float2 &lz, const float4 *__restrict__ apt,
                                               const float4 *__restrict__ aph, const int (&pt)[KPL],
                                               const float2 (&npx)[KPL], const float2 (&npy)[KPL],
                                               const float2 (&npz)[KPL], const PairConst &c, PairAccP<KPL> &acc)
{
  const float2 lj01 = f2(c.lj01), lj0 = f2(c.lj0), one = f2(1.0f), inv_el1 = f2(c.inv_el1);
  const float2 za = f2(-0.5f * kLog2e), zb = f2(6.0f * kLog2e);
#pragma unroll
  for (int j = 0; j < KPL; ++j) {
    const int e = i * kTabCols + pt[j];
    const float4 ta = apt[2 * e], tb = apt[GD_AT(2 * e + 1, 2 * npairs * kTabCols, kSiteApt)];
    const float2 dx = __fadd2_rn(lx, npx[j]), dy = __fadd2_rn(ly, npy[j]), dz = __fadd2_rn(lz, npz[j]);
    const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    const float2 r = make_float2(rsqrt_approx(d2.x), rsqrt_approx(d2.y));
    const float2 d = __fmul2_rn(d2, r);
    const float2 d3 = __fmul2_rn(d2, d);
    const float2 d6 = __fmul2_rn(d3, d3);
    const float2 den = __ffma2_rn(__fmul2_rn(d6, d3), make_float2(ta.x, ta.y), __ffma2_rn(lj01, d2, lj0));
    const float2 num = __ffma2_rn(make_float2(ta.z, ta.w), d3, one);
    acc.vdw = __ffma2_rn(num, make_float2(rcp_approx(den.x), rcp_approx(den.y)), acc.vdw);
    float2 g = __fmul2_rn(r, inv_el1);
    if constexpr (DEEP) {
      const float2 near = __ffma2_rn(d2, __ffma2_rn(f2(c.eb), d, f2(c.ea)), f2(c.el0));
      g.x = d2.x < c.ed2 ? near.x : g.x;
      g.y = d2.y < c.ed2 ? near.y : g.y;
    } else {
      if (d2.x < c.ed2) g.x = __fmaf_rn(d2.x, __fmaf_rn(c.eb, d.x, c.ea), c.el0);
      if (d2.y < c.ed2) g.y = __fmaf_rn(d2.y, __fmaf_rn(c.eb, d.y, c.ea), c.el0);
    }
    acc.ele[j] = __ffma2_rn(lig[GD_AT(i, npairs, kSiteLig)].q, g, acc.ele[j]);
    const float2 dmp = __fadd2_rn(d, make_float2(tb.x, tb.y));
    const float2 z = __fmul2_rn(__ffma2_rn(za, d, zb), dmp);
    const float2 e1 = __fadd2_rn(make_float2(ex2_approx(z.x), ex2_approx(z.y)), one);
    acc.pmf = __ffma2_rn(make_float2(tb.z, tb.w), make_float2(rcp_approx(e1.x), rcp_approx(e1.y)), acc.pmf);
    if constexpr (HDB) {
      const float4 th = aph[GD_AT(e, npairs * kTabCols, kSiteAph)];
      const float2 hb = __ffma2_rn(d, make_float2(th.x, th.y), make_float2(th.z, th.w));
      const float2 hh = __fmul2_rn(hb, hb);
      acc.hdb = __ffma2_rn(make_float2(th.x, th.y), make_float2(ex2_approx(-hh.x), ex2_approx(-hh.y)), acc.hdb);
    }
  }
}

// Pass 1 over the 32 KPL points from `row`: (vdw, ele, pmf, hdb) per lane.
// Lane i holds points row + i + 32 j; a warp reduction gives the point types
// present, and the hydrogen-bond code runs only for the atom pairs that need it
// (where it is not needed, every value it would add is 0).  DEEP: the pairs up
// to the last that needs it run with the term and the others without, in two
// loops without a branch (the near-field electrostatics selected rather than
// branched to), unrolled so that the chains of the points and of two pairs
// overlap: for a warp that has the scheduler almost to itself.
template <int KPL, bool DEEP>
__device__ __forceinline__ float4 pass1_row(const LigPair *lp, int npairs, int row, int P, const float4 *__restrict__ pos,
                                            const float2 *__restrict__ aux, const float4 *__restrict__ apt,
                                            const float4 *__restrict__ aph, const int4 *__restrict__ ahd,
                                            const PairConst &kc)
{
  const int lane = lane_id();
  float2 npx[KPL], npy[KPL], npz[KPL];
  int pt[KPL];
  uint32_t ptbits = 0u;
#pragma unroll
  for (int j = 0; j < KPL; ++j) {
    const int p = GD_AT(row + 32 * j + lane, P, kSitePos);
    const float4 q = pos[p];
    npx[j] = f2(-q.x);
    npy[j] = f2(-q.y);
    npz[j] = f2(-q.z);
    pt[j] = __float_as_int(aux[p].y);
    ptbits |= 1u << pt[j];
  }
  ptbits = __reduce_or_sync(0xffffffffu, ptbits);
  PairAccP<KPL> acc;
  acc.vdw = acc.pmf = acc.hdb = f2(0.0f);
#pragma unroll
  for (int j = 0; j < KPL; ++j) acc.ele[j] = f2(0.0f);
  if constexpr (DEEP) {
    int nh = 0;  // pairs [0, nh) with the hydrogen-bond term
    for (int i = lane; i < npairs; i += 32)
      if ((uint32_t)ahd[GD_AT(i, npairs, kSiteAhd)].x & ptbits) nh = i + 1;
    nh = __reduce_max_sync(0xffffffffu, nh);
    int i = 0;
#pragma unroll 2
    for (; i < nh; ++i) {
      const float4 l01 = *reinterpret_cast<const float4 *>(&lp[GD_AT(i, npairs, kSiteLig)].x);
      pair_atom_pair<KPL, true, true>(lp, i GD_CHECK_ARG(npairs), make_float2(l01.x, l01.y), make_float2(l01.z, l01.w),
                                      lp[i].z, apt, aph, pt, npx, npy, npz, kc, acc);
    }
#pragma unroll 2
    for (; i < npairs; ++i) {
      const float4 l01 = *reinterpret_cast<const float4 *>(&lp[GD_AT(i, npairs, kSiteLig)].x);
      pair_atom_pair<KPL, false, true>(lp, i GD_CHECK_ARG(npairs), make_float2(l01.x, l01.y), make_float2(l01.z, l01.w),
                                       lp[i].z, apt, aph, pt, npx, npy, npz, kc, acc);
    }
  } else {
    for (int i = 0; i < npairs; ++i) {
      const int2 fl = *reinterpret_cast<const int2 *>(&ahd[GD_AT(i, npairs, kSiteAhd)].x);
      const bool any_hdb = ((uint32_t)fl.x & ptbits) != 0u;
      const float4 l01 = *reinterpret_cast<const float4 *>(&lp[GD_AT(i, npairs, kSiteLig)].x);
      const float2 lx = make_float2(l01.x, l01.y), ly = make_float2(l01.z, l01.w), lz = lp[i].z;
      if (any_hdb)
        pair_atom_pair<KPL, true, false>(lp, i GD_CHECK_ARG(npairs), lx, ly, lz, apt, aph, pt, npx, npy, npz, kc, acc);
      else
        pair_atom_pair<KPL, false, false>(lp, i GD_CHECK_ARG(npairs), lx, ly, lz, apt, aph, pt, npx, npy, npz, kc, acc);
    }
  }
  float4 h;
  h.y = 0.0f;
#pragma unroll
  for (int j = 0; j < KPL; ++j)
    // the point charges are read again here rather than held through the atom loop
    h.y = fma_(pos[row + 32 * j + lane].w, add_(acc.ele[j].x, acc.ele[j].y), h.y);
  h.x = add_(acc.vdw.x, acc.vdw.y);
  h.z = add_(acc.pmf.x, acc.pmf.y);
  h.w = add_(acc.hdb.x, acc.hdb.y);
  return h;
}

// Component c of pass1_row<4>'s sums, alone: the terms of atoms c, c + 2, ... (of
// the atom pairs) against the 128 points from `row`, in scalar arithmetic, the
// same operations in the same order; a team joins the two components to pass1_row's
// sums where it combines its units.  Two warps then share a row, where a team has warps to spare.
struct HalfRow {
  float vdw, pmf, hdb, ele[4];
};

template <bool HDB>
__device__ __forceinline__ void pair_atom(const float *__restrict__ lf, int e0, const float *__restrict__ apt,
                                          const float *__restrict__ aph, const int (&pt)[4], const float (&npx)[4],
                                          const float (&npy)[4], const float (&npz)[4], const PairConst &c, HalfRow &acc)
{
  const float lx = lf[0], ly = lf[2], lz = lf[4], lq = lf[6];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int e = e0 + pt[j];
    const float *ta = apt + 8 * e;
    const float dx = add_(lx, npx[j]), dy = add_(ly, npy[j]), dz = add_(lz, npz[j]);
    const float d2 = dist2(dx, dy, dz);
    const float r = rsqrt_approx(d2);
    const float d = mul_(d2, r);
    const float d3 = mul_(d2, d);
    const float d6 = mul_(d3, d3);
    const float den = fma_(mul_(d6, d3), ta[0], fma_(c.lj01, d2, c.lj0));
    const float num = fma_(ta[2], d3, 1.0f);
    acc.vdw = fma_(num, rcp_approx(den), acc.vdw);
    const float near = fma_(d2, fma_(c.eb, d, c.ea), c.el0);
    const float g = d2 < c.ed2 ? near : mul_(r, c.inv_el1);
    acc.ele[j] = fma_(lq, g, acc.ele[j]);
    const float z = mul_(fma_(-0.5f * kLog2e, d, 6.0f * kLog2e), add_(d, ta[4]));
    acc.pmf = fma_(ta[6], rcp_approx(add_(ex2_approx(z), 1.0f)), acc.pmf);
    if constexpr (HDB) {
      const float *th = aph + 4 * e;
      const float hb = fma_(d, th[0], th[2]);
      acc.hdb = fma_(th[0], ex2_approx(-mul_(hb, hb)), acc.hdb);
    }
  }
}

__device__ __forceinline__ HalfRow pass1_half(const LigPair *lp, int npairs, int c, int row, int P,
                                              const float4 *__restrict__ pos, const float2 *__restrict__ aux,
                                              const float4 *__restrict__ apt, const float4 *__restrict__ aph,
                                              const int4 *__restrict__ ahd, const PairConst &kc)
{
  const int lane = lane_id();
  float npx[4], npy[4], npz[4];
  int pt[4];
  uint32_t ptbits = 0u;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int p = GD_AT(row + 32 * j + lane, P, kSitePos);
    const float4 q = pos[p];
    npx[j] = -q.x;
    npy[j] = -q.y;
    npz[j] = -q.z;
    pt[j] = __float_as_int(aux[p].y);
    ptbits |= 1u << pt[j];
  }
  ptbits = __reduce_or_sync(0xffffffffu, ptbits);
  int nh = 0;  // pairs [0, nh) with the hydrogen-bond term
  for (int i = lane; i < npairs; i += 32)
    if ((uint32_t)ahd[GD_AT(i, npairs, kSiteAhd)].x & ptbits) nh = i + 1;
  nh = __reduce_max_sync(0xffffffffu, nh);
  HalfRow acc{0.f, 0.f, 0.f, {0.f, 0.f, 0.f, 0.f}};
  const float *lf = reinterpret_cast<const float *>(lp) + c;
  const float *ta = reinterpret_cast<const float *>(apt) + c, *th = reinterpret_cast<const float *>(aph) + c;
  int i = 0;
#pragma unroll 2
  for (; i < nh; ++i) pair_atom<true>(lf + 8 * i, i * kTabCols, ta, th, pt, npx, npy, npz, kc, acc);
#pragma unroll 2
  for (; i < npairs; ++i) pair_atom<false>(lf + 8 * i, i * kTabCols, ta, th, pt, npx, npy, npz, kc, acc);
  return acc;
}

// The running sums of pass 1 over the rows, in row order: compensated for the
// three dense terms with the FP32-Kahan policy (hdb is a short, sparse sum).
template <int PREC>
struct RowSums {
  using T = RealOf<PREC>;
  T s[4] = {0, 0, 0, 0};  // vdw, ele, pmf, hdb
  float c[3] = {0.f, 0.f, 0.f};
  __device__ __forceinline__ void add(int term, T x)
  {
    if constexpr (PREC == kFP32Kahan) {
      if (term < 3) {
        kahan_add(s[term], c[term], x);
        return;
      }
    }
    s[term] = add_(s[term], x);
  }
  // the sum over the warp's lanes
  __device__ __forceinline__ T total(int term) const
  {
    if constexpr (PREC == kFP32Kahan)
      if (term < 3) return warp_sum_comp(s[term], c[term]);
    return warp_sum(s[term]);
  }
};

// ------------------------------------------------------ pair loop, FP64 --
// Reciprocal in FP64: the PTX approximation (an error of up to 1e-6) and one step
// of the third-order Newton (Halley) iteration, which cubes that: the rounding of the
// last operation is what remains (within 1.12e-16 relative).  x positive, normal and
// finite, as every argument below is.
__device__ __forceinline__ double rcp64(double x)
{
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma_(-x, y, 1.0);
  return fma_(y, fma_(e, e, e), y);
}
// Square root d of x and half the reciprocal of it, h, in FP64: from the PTX approximation
// y the pair (x y, y / 2), corrected by one third-order step (Goldschmidt's form of
// the iteration, whose error e undoes half the rounding of x y: d is within 1.7e-16
// relative, rms 4.9e-17, where x (1 / sqrt(x)) has 2.2e-16 and 7.0e-17 and sqrt() 1.1e-16
// and 4.4e-17).  x positive, normal and finite.
__device__ __forceinline__ void sqrt64(double x, double &d, double &h)
{
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h0 = __hiloint2double(__double2hiint(y) - 0x100000, __double2loint(y));  // y / 2
  const double g = mul_(x, y);
  const double e = fma_(-g, h0, 0.5);
  const double t = fma_(mul_(1.5, e), e, e);
  h = fma_(h0, t, h0);
  d = fma_(g, t, g);
}

constexpr int kExpTab = 256;

// Entry j of the exponential's table: 2^(j / 256) as the sum of two doubles, tab[j] and
// tab[256 + j], from the product of the 2^(2^b / 256) of j's bits (an error of about 1e-31).
__device__ __forceinline__ void exp_table_entry(double *tab, int j)
{
  constexpr double kPow[8][2] = {{1.0027112750502025, -3.6366159286922639e-17}, {1.0054299011128027, 9.4991865354550318e-17},
                                 {1.0108892860517005, -1.5234778603368577e-17}, {1.0218971486541166, 5.1092250289734439e-17},
                                 {1.0442737824274138, 8.5518897055379649e-17}, {1.0905077326652577, -3.0467820798124711e-17},
                                 {1.189207115002721, 3.9820152314656461e-17}, {1.4142135623730951, -9.6672933134529135e-17}};
  double hi = 1.0, lo = 0.0;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    if (!((j >> b) & 1)) continue;
    const double p = mul_(hi, kPow[b][0]);
    const double e = fma_(hi, kPow[b][0], -p) + fma_(hi, kPow[b][1], mul_(lo, kPow[b][0]));
    hi = add_(p, e);
    lo = sub_(e, sub_(hi, p));
  }
  tab[j] = hi;
  tab[kExpTab + j] = lo;
}

// exp(x) in FP64 after Tang (Table-driven implementation of the exponential
// function in IEEE floating-point arithmetic, ACM TOMS 15, 1989): x = (256 m + j)
// ln2/256 + r, |r| <= ln2/512 = a, exp(x) = 2^m 2^(j/256) exp(r), exp(r) - 1 from its
// Taylor series to r^4 with the coefficient of r^3 raised by (3/4) a^2 / 120, which
// takes up most of the fifth power (remainder below 1e-17), 2^(j/256) from tab, with its
// second part (LOW) or without.  Within 1.3e-16 (2.4e-16) relative of the exponential on
// [-700, 700]; CUDA's exp() was measured within 1.36e-16.  The pmf term takes the
// form without: its factor 1 / (1 + exp(z)) carries |z| times the rounding of z, 3.8e-16
// rms, and the second part changes that by a thousandth.  Beyond the range 0 and 2^1000,
// whose reciprocals act as those of exp() would; NaN stays NaN.
template <bool LOW>
__device__ __forceinline__ double exp64(double x, const double *tab)
{
  constexpr double kMagic = 6755399441055744.0;  // 1.5 2^52: the nearest integer in the low word
  constexpr double kA = 0.6931471805599453 / 512.0;
  const double k = fma_(x, 8 * 46.16624130844683, kMagic);
  const int n = __double2loint(k);
  const double kn = sub_(k, kMagic);
  const double r = fma_(kn, -7.247021293269686e-19 / 8, fma_(kn, -0.02166084939249829 / 8, x));
  double p = fma_(r, 1.0 / 24.0, 1.0 / 6.0 + 0.75 * kA * kA / 120.0);
  p = fma_(p, r, 0.5);
  const double q = fma_(mul_(p, r), r, r);  // exp(r) - 1
  const int j = n & (kExpTab - 1);
  const double t = tab[j], v = LOW ? add_(t, fma_(t, q, tab[kExpTab + j])) : fma_(t, q, t);
  int hi = __double2hiint(v) + ((n >> 8) << 20), lo = __double2loint(v);
  const int xh = __double2hiint(x), mag = xh & 0x7fffffff;
  if (mag > 0x4085e000) {  // |x| > 700, infinite or NaN
    hi = mag > 0x7ff00000 ? 0x7ff80000 : xh < 0 ? 0 : 0x7e700000;
    lo = 0;
  }
  return __hiloint2double(hi, lo);
}

// Per work item, the FP64 kernel's (ligand type group, point type) entries in
// shared memory: pk = (1/p1a, -p2a), pf = (-pmf0, pmf1, hdb0, hdb1), the
// hydrogen-bond entries zero where hdb0 <= 0.1; and the exponential's table.
// Padding point types get 1/p1a = 1e30 and 0 else: at their distance (over 1e3)
// their Lennard-Jones term is below 1e-57, the others exactly 0.
__device__ __forceinline__ void build_pair_tables64(const DevJob &J, const int2 *lg, double2 *pk, float4 *pf, double *tab)
{
  const int L = J.natom;
  for (int j = threadIdx.x; j < kExpTab; j += blockDim.x) exp_table_entry(tab, j);
  int g = 0;
  for (int a = 0; a < L; ++g) {
    const int lt = GD_AT(lg[GD_AT(a, L, kSiteLgrp)].x, kLigTypes, kSiteTab);
    for (int pt = threadIdx.x; pt < kTabCols; pt += blockDim.x) {
      const float4 r = J.ref4[lt * kTabCols + pt], t = J.par->tab4[lt][pt];
      const bool real = pt < kPadType;
      pk[g * kTabCols + pt] = real ? make_double2(1.0 / (double)r.x, -(double)r.y) : make_double2(1.0e30, 0.0);
      pf[g * kTabCols + pt] = real ? make_float4(t.z, t.w, r.z, r.w) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    a = lg[a].y;
  }
}

// Terms of the atoms [a, aend) of one type against the lane's two points, the
// reference's formulas with the Lennard-Jones term divided through by p1 (as in
// FP32; p = d^3 / p1a in numerator and denominator, so that its rounding cancels where
// the term decays), which leaves one square root, two reciprocals and one exponential
// per pair.  Bound by the FP64 pipe (2.04 cycles a warp operation and scheduler, 45 a
// pair) and the issue of the ~30 others.  2048 poses of 64 atoms x 3000 points: 2.73 ms
// with CUDA's rsqrt, __drcp_rn and exp, 2.16 with the Newton steps and an exponential
// from a table of 32, 2.03 with one of 256 and the near field told by d^2, 2.06 in the
// forms here, which are no less exact than the reference's in double (8,300 poses against
// 113-bit arithmetic, rms error of the terms vdw, ele, pmf, hdb, hpc relative to their mean:
// 3.65, 8.50, 0.58, 4.35 and 2.27e-16; formulas as written with CUDA's functions 3.69, 9.13,
// 0.58, 4.39 and 2.43e-16; d as x (1 / sqrt(x)) and the exponential without its table's
// second part 4.57e-16 for hdb).  The table's second part for the pmf term's exponential
// too takes 6 % more, d corrected by its remainder 3 %.  1e-300 keeps d > 0 where a point
// and an atom coincide.
template <bool HDB>
__device__ __forceinline__ void pair_atoms64(const V4<double> *lig, int a, int aend, int L, const double (&px)[2],
                                             const double (&py)[2], const double (&pz)[2], const double2 (&k)[2],
                                             const float4 (&f)[2], const PairConst64 &c, double (&vdw)[2],
                                             double (&ele)[2], double (&pmf)[2], double (&hdb)[2])
{
#pragma unroll 1
  for (; a < aend; ++a) {
    const V4<double> la = lig[GD_AT(a, L, kSiteLig)];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const double dx = sub_(la.x, px[j]), dy = sub_(la.y, py[j]), dz = sub_(la.z, pz[j]);
      const double d2 = fma_(dx, dx, fma_(dy, dy, fma_(dz, dz, 1.0e-300)));
      double d, h;
      sqrt64(d2, d, h);
      const double p = mul_(mul_(d2, d), k[j].x);
      double d6 = mul_(mul_(d2, d2), d2);
      // at most 2^450 (from 4e22 A on, where the term is below 1e-130): den stays finite
      d6 = __hiloint2double(min(__double2hiint(d6), 0x5c100000), __double2loint(d6));
      const double den = fma_(d6, p, fma_(c.lj01, d2, c.lj0));
      vdw[j] = fma_(fma_(k[j].y, p, 1.0), rcp64(den), vdw[j]);
      const double g = d2 < c.ed2 ? fma_(d2, fma_(c.eb, d, c.ea), c.el0) : mul_(h, c.inv_el1);
      ele[j] = fma_(la.w, g, ele[j]);
      const double e1 = add_(1.0, exp64<false>(mul_(fma_(-0.5, d, 6.0), add_(d, (double)f[j].x)), c.tab));
      pmf[j] = fma_((double)f[j].y, rcp64(e1), pmf[j]);
      if constexpr (HDB) {
        const double h3 = mul_(sub_(d, (double)f[j].z), (double)f[j].w);
        hdb[j] = fma_((double)f[j].w, exp64<true>(mul_(mul_(-0.5, h3), h3), c.tab), hdb[j]);
      }
    }
  }
}

// Pass 1 over the 128 points from `row` in FP64, two points per lane at a time.
__device__ __forceinline__ void pass1_row64(const V4<double> *lig, int L, const int2 *lgrp, const DevParams *par,
                                            const double2 *pk, const float4 *pf, const double *tab, int row, int P,
                                            const float4 *pos, const float2 *aux, double (&h)[4])
{
  const int lane = lane_id();
  PairConst64 c;
  c.lj0 = par->lj0;
  c.lj01 = mul_(c.lj0, (double)par->lj1);
  c.el0 = par->el0;
  const double el1 = par->el1;
  c.ea = mul_(mul_((double)par->a1, el1), el1);
  c.eb = mul_(mul_(mul_((double)par->b1, el1), el1), el1);
  c.inv_el1 = mul_(2.0, __drcp_rn(el1));  // of half of 1/d
  c.ed2 = el1 > 0.0 ? __drcp_rn(mul_(el1, el1)) : INFINITY;  // el1 d < 1
  c.tab = tab;
  double vdw[2] = {0, 0}, pmf[2] = {0, 0}, hdb[2] = {0, 0}, qe = 0;
#pragma unroll 1
  for (int sub = 0; sub < kRowPoints; sub += 64) {
    double px[2], py[2], pz[2], pe[2], ele[2] = {0, 0};
    int pt[2];
    uint32_t ptbits = 0u;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int p = GD_AT(row + sub + 32 * j + lane, P, kSitePos);
      const float4 q = pos[p];
      px[j] = q.x; py[j] = q.y; pz[j] = q.z; pe[j] = q.w;
      pt[j] = __float_as_int(aux[p].y);
      ptbits |= 1u << pt[j];
    }
    ptbits = __reduce_or_sync(0xffffffffu, ptbits);
    int g = 0;
    for (int a = 0; a < L; ++g) {
      const int2 grp = lgrp[GD_AT(a, L, kSiteLgrp)];
      const int aend = grp.y;
      double2 k[2];
      float4 f[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        k[j] = pk[g * kTabCols + pt[j]];
        f[j] = pf[g * kTabCols + pt[j]];
      }
      if (par->hdbmask[GD_AT(grp.x, kLigTypes, kSiteTab)] & ptbits)
        pair_atoms64<true>(lig, a, aend, L, px, py, pz, k, f, c, vdw, ele, pmf, hdb);
      else
        pair_atoms64<false>(lig, a, aend, L, px, py, pz, k, f, c, vdw, ele, pmf, hdb);
      a = aend;
    }
    qe = fma_(pe[1], ele[1], fma_(pe[0], ele[0], qe));
  }
  h[0] = add_(vdw[0], vdw[1]);
  h[1] = qe;
  h[2] = add_(pmf[0], pmf[1]);
  h[3] = add_(hdb[0], hdb[1]);
}

// -------------------------------------------------- hydrophobic contact --
// Pass 2 (energy_prt_v1.cu:42-49) visits only the 64-point rows holding cdc == 1
// points (placed first); 64 whatever pass 1 uses, so that the last row carries
// at most 63 others (hpp 0).
__device__ __forceinline__ int contact_rows(const DevJob &J, int iprt)
{
  return (J.ncdc[iprt] + kHalfPoints - 1) / kHalfPoints * kHalfPoints;
}

// Contact sums of the AB atoms from a0 over the rows row0, row0 + rstep, ...  The polynomial
// 1 - 3.5x + 4.5x^2 - 2.5x^3 + 0.5x^4 (x = d^2/81) is (1-x)^3 (1-x/2), i.e.
// (y^3 + y^4) / 2 with y = 1 - x; clamping y at 0 applies the d^2 <= 81 cut-off;
// the loop sums hpp y^2 (y + y^2), halved exactly at the end.  The AB sums are
// reduced across the warp together (each butterfly step halves the sums a lane
// carries: it keeps the half its lane bit selects and adds its partner's copy
// of it): lane l ends with the sum of atom a0 + l / (32 / AB).
template <int PREC, int AB>
__device__ __forceinline__ RealOf<PREC> contact_block(const LigOf<PREC> *lig, int L, int a0, int row0, int rstep,
                                                      int rows, const float4 *__restrict__ pos,
                                                      const float2 *__restrict__ aux, int P)
{
  using T = RealOf<PREC>;
  const int lane = lane_id();
  T v[AB];
  if constexpr (PREC != kFP64) {
    const float2 one = f2(1.0f), c1 = f2(-1.0f / 81.0f);
    float2 h2[AB / 2];
#pragma unroll
    for (int k = 0; k < AB / 2; ++k) h2[k] = f2(0.0f);
    for (int row = row0; row < rows; row += rstep) {
      float2 npx[2], npy[2], npz[2], ph2[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int p = GD_AT(row + 32 * j + lane, P, kSitePos);
        const float4 q = pos[p];
        npx[j] = f2(-q.x);
        npy[j] = f2(-q.y);
        npz[j] = f2(-q.z);
        ph2[j] = f2(aux[p].x);
      }
#pragma unroll
      for (int k = 0; k < AB / 2; ++k) {
        const int a = a0 + 2 * k;
        if (a >= L) break;
        const LigPair la = lig[GD_AT(a >> 1, (L + 1) >> 1, kSiteLig)];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 dx = __fadd2_rn(la.x, npx[j]), dy = __fadd2_rn(la.y, npy[j]), dz = __fadd2_rn(la.z, npz[j]);
          const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
          float2 y = __ffma2_rn(d2, c1, one);
          y.x = fmaxf(y.x, 0.0f);
          y.y = fmaxf(y.y, 0.0f);
          const float2 yy = __fmul2_rn(y, y);
          const float2 w = __fmul2_rn(yy, __fadd2_rn(y, yy));
          h2[k] = __ffma2_rn(ph2[j], w, h2[k]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < AB / 2; ++k) {
      v[2 * k] = 0.5f * h2[k].x;
      v[2 * k + 1] = 0.5f * h2[k].y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < AB; ++k) v[k] = 0;
    for (int row = row0; row < rows; row += rstep) {
#pragma unroll 1
      for (int j = 0; j < 2; ++j) {
        const int p = GD_AT(row + 32 * j + lane, P, kSitePos);
        const float4 q = pos[p];
        const double px = q.x, py = q.y, pz = q.z, ph = aux[p].x;
#pragma unroll
        for (int k = 0; k < AB; ++k) {
          const int a = a0 + k;
          if (a >= L) break;
          const V4<double> la = lig[GD_AT(a, L, kSiteLig)];
          const double d2 = dist2(sub_(la.x, px), sub_(la.y, py), sub_(la.z, pz));
          const double y = fmax(fma_(d2, -1.0 / 81.0, 1.0), 0.0);
          v[k] = fma_(ph, mul_(mul_(mul_(y, y), y), fma_(d2, -0.5 / 81.0, 1.0)), v[k]);
        }
      }
    }
  }
#pragma unroll
  for (int n = AB, off = 16; n > 1; n >>= 1, off >>= 1) {
    const bool hi = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const T keep = hi ? v[n / 2 + i] : v[i], give = hi ? v[i] : v[n / 2 + i];
      v[i] = add_(keep, __shfl_xor_sync(0xffffffffu, give, off));
    }
  }
#pragma unroll
  for (int off = 16 / AB; off > 0; off >>= 1) v[0] = add_(v[0], __shfl_xor_sync(0xffffffffu, v[0], off));
  return v[0];
}

// The restraint on atom a's contact sum S (energy_prt_v1.cu:162-169).
template <typename T>
__device__ __forceinline__ T contact_restraint(const DevParams *par, const int2 *lgrp, int a, int L, T S)
{
  const int lt = GD_AT(lgrp[GD_AT(a, L, kSiteLgrp)].x, kLigTypes, kSiteTab);
  const T h = sub_(S, (T)par->hpl0[lt]) / (T)par->hpl1[lt];
  return fma_(mul_((T)0.5, h), h, -(T)par->hpl2[lt]);
}

// A lane's share of one chunk of a walk: what the one-warp kernel adds to the
// lane's sum as fma(x, w, sum).
template <typename T>
struct WalkTerm {
  T x, w;
};

// ------------------------------------------------- pocket-specific term --
// Cell k of the term's list (energy_prt_v1.cu:109-115), the conformation's
// non-zero cells (point p, ligand type t, value; only types the ligand has)
// ordered by type: counts the atoms of type t (the contiguous range [beg, end)
// of the type-grouped ligand) with d - pmf0 <= 0; in FP32 with the operations
// of the pair loop for d.  A cell is two independent 16-byte loads.
template <int PREC>
__device__ __forceinline__ WalkTerm<RealOf<PREC>> psp_cell(const int4 *cell, int stride, int L, const LigOf<PREC> *lig,
                                                           int k)
{
  using T = RealOf<PREC>;
  const int4 c0 = __ldg(cell + 2 * GD_AT(k, stride, kSitePsp));
  const int4 c1 = __ldg(cell + 2 * k + 1);
  const int beg = c1.x & 0xffff, end = c1.x >> 16;
  const T thr = (T)__int_as_float(c1.y);
  const T nx = -(T)__int_as_float(c0.x), ny = -(T)__int_as_float(c0.y), nz = -(T)__int_as_float(c0.z);
  int hits = 0;
  for (int a = beg; a < end; ++a) {
    const V4<T> la = atom_at(lig, GD_AT(a, L, kSiteLig));
    const T d2 = dist2(add_(la.x, nx), add_(la.y, ny), add_(la.z, nz));
    T d;
    if constexpr (PREC == kFP64) d = sqrt(d2);
    else d = mul_(d2, rsqrt_approx(d2));
    hits += add_(d, thr) <= (T)0 ? 1 : 0;
  }
  // (the FP32 loop over these cells has always multiplied; the others added the value of a hit only)
  if (PREC == kFP64 && hits == 0) return {0, 0};
  return {(T)hits, (T)__int_as_float(c0.w)};
}

// The same of a 4-byte cell (pack_cell4), gathered through it.
template <int PREC>
__device__ __forceinline__ WalkTerm<RealOf<PREC>> psp_cell4(const DevJob &J, int iprt, const LigOf<PREC> *lig, int k)
{
  using T = RealOf<PREC>;
  const int c = J.pcell4[(size_t)iprt * J.pcell_stride + GD_AT(k, J.pcell_stride, kSitePsp)];
  const int j = c & 2047, t = (c >> 11) & 31, L = J.natom;
  const size_t p = (size_t)iprt * J.npoint_pad + j;
  const float4 q = J.pos[p];
  const T thr = (T)J.par->tab4[t][__float_as_int(J.aux[p].y)].z;
  const T nx = -(T)q.x, ny = -(T)q.y, nz = -(T)q.z;
  const int range = J.trange[t];
  int hits = 0;
  for (int a = range & 0xffff; a < range >> 16; ++a) {
    const V4<T> la = atom_at(lig, GD_AT(a, L, kSiteLig));
    const T d2 = dist2(add_(la.x, nx), add_(la.y, ny), add_(la.z, nz));
    T d;
    if constexpr (PREC == kFP64) d = sqrt(d2);
    else d = mul_(d2, rsqrt_approx(d2));
    hits += add_(d, thr) <= (T)0 ? 1 : 0;
  }
  // a cell without a hit adds nothing, be its value infinite or NaN
  if (hits == 0) return {0, 0};
  return {(T)hits, (T)J.psp_table[t * GD_MAXPRO + (c >> 16)]};
}

// The chunks c0, c0 + cstep, ... of 32 cells in turn (C4: 4-byte cells).
template <int PREC, bool C4>
__device__ __forceinline__ RealOf<PREC> psp_walk(const DevJob &J, int iprt, const LigOf<PREC> *lig, int c0, int cstep)
{
  using T = RealOf<PREC>;
  const int4 *cell = J.pcell + (size_t)iprt * J.pcell_stride * 2;
  const int n = J.pcell_cnt[iprt], L = J.natom, stride = J.pcell_stride;
  T acc = 0;
  for (int k = 32 * c0 + lane_id(); k < n; k += 32 * cstep) {
    WalkTerm<T> t;
    if constexpr (C4) t = psp_cell4<PREC>(J, iprt, lig, k);
    else t = psp_cell<PREC>(cell, stride, L, lig, k);
    acc = fma_(t.x, t.w, acc);
  }
  return acc;
}

// ---------------------------------------------------------------- KDE --
// Slot q of the term (energy_kde_v1.cu:183-274), a KDE point of a type the
// ligand has: the sum of exp(kde2 d^2) over the atoms of its type group and the
// weight 1/(points of the type): every lane busy, one coalesced pair of loads
// per slot, no division in FP32.
template <int PREC>
__device__ __forceinline__ WalkTerm<RealOf<PREC>> kde_slot(const int4 *slot, int n, int L, RealOf<PREC> k2,
                                                           const LigOf<PREC> *lig, int q)
{
  using T = RealOf<PREC>;
  const int4 c0 = __ldg(slot + 2 * GD_AT(q, n, kSiteKde));
  const int4 c1 = __ldg(slot + 2 * q + 1);
  const T qx = (T)__int_as_float(c0.x), qy = (T)__int_as_float(c0.y), qz = (T)__int_as_float(c0.z);
  T sk = 0;
  const int end = c1.x >> 16;
  for (int b = c1.x & 0xffff; b < end; ++b) {
    const V4<T> la = atom_at(lig, GD_AT(b, L, kSiteLig));
    const T d2 = dist2_xyz(sub_(la.x, qx), sub_(la.y, qy), sub_(la.z, qz));
    if constexpr (PREC == kFP64) sk = add_(sk, exp(mul_(k2, d2)));
    else sk = add_(sk, ex2_approx(mul_(k2, d2)));
  }
  if constexpr (PREC == kFP64) return {sk / (double)c1.y, 1.0};
  else return {sk, __int_as_float(c0.w)};
}

template <int PREC>
__device__ __forceinline__ RealOf<PREC> kde_exponent(const DevParams *par)
{
  if constexpr (PREC == kFP64) return (double)par->kde2;
  else return mul_(par->kde2, kLog2e);
}

// The chunks c0, c0 + cstep, ... of 32 slots in turn.
template <int PREC>
__device__ __forceinline__ RealOf<PREC> kde_walk(const DevJob &J, const DevParams *par, const LigOf<PREC> *lig, int c0,
                                                 int cstep)
{
  using T = RealOf<PREC>;
  const T k2 = kde_exponent<PREC>(par);
  const int4 *slot = J.kslot;
  const int n = J.nkslot, cap = J.nkde, L = J.natom;
  T acc = 0;
  for (int q = 32 * c0 + lane_id(); q < n; q += 32 * cstep) {
    const WalkTerm<T> t = kde_slot<PREC>(slot, cap, L, k2, lig, q);
    acc = fma_(t.x, t.w, acc);
  }
  return acc;
}

// ---------------------------------------------------------------- MCS --
// Sums over the templates of tcc * rmsd (energy_mcs_v1.cu:277-320), by one warp,
// in V shares: up to 16 templates the templates v, v + V, ..., else the runs of
// 32 templates v, v + V, ...  out[v]: share v's sum (the return value: share 0's).
template <int PREC>
__device__ __forceinline__ RealOf<PREC> mcs_sums(const DevJob &J, const LigOf<PREC> *lig, int V, RealOf<PREC> *out)
{
  using T = RealOf<PREC>;
  const int lane = lane_id(), M = J.nmcs, L = J.natom;
  const float4 *mcs = J.mcs;
  // up to 16 templates: two half-warps share each (its even and odd atoms)
  const bool halves = M <= 16;
  const int step = halves ? 2 : 1, m_of = halves ? lane & 15 : lane, first = halves ? lane >> 4 : 0;
  T x0 = 0;
  for (int v = 0; v < (halves ? 1 : V); ++v) {
    T macc = 0;
    for (int m0 = halves ? 0 : 32 * v; m0 < M; m0 += 32 * (halves ? 1 : V)) {
      const int m = m0 + m_of;
      T s = 0;
      int n = 0;
      if (m < M) {
        // an atom the template does not place adds 0
#pragma unroll 4
        for (int a = first; a < L; a += step) {
          const float4 q = mcs[GD_AT((size_t)a * M + m, (size_t)L * M, kSiteMcs)];
          const V4<T> la = atom_at(lig, a);
          const T d2 = dist2_xyz(sub_(la.x, (T)q.x), sub_(la.y, (T)q.y), sub_(la.z, (T)q.z));
          s = add_(s, q.w != 0.0f ? d2 : (T)0);
          n += q.w != 0.0f;
        }
      }
      if (halves) {
        s = add_(s, __shfl_xor_sync(0xffffffffu, s, 16));
        n += __shfl_xor_sync(0xffffffffu, n, 16);
      }
      if (m < M && first == 0) macc = fma_((T)J.tcc[GD_AT(m, M, kSiteTcc)], (T)sqrt(s / (T)n), macc);
    }
    if (V == 1) return warp_sum(macc);
    for (int w = halves ? 0 : v; w < (halves ? V : v + 1); ++w) {
      const T x = warp_sum(halves && m_of % V != w ? (T)0 : macc);
      if (lane == 0) out[w] = x;
      if (w == 0) x0 = x;
    }
  }
  return x0;
}

// ------------------------------------------------------------- the end --
// Squared distance of the ligand centre to the pocket centre,
// kernel_cuda_l1_montecarlo.cu:439-454; lane k < 6 holds movematrix[k] in pm.
template <typename T>
__device__ __forceinline__ T centre_dist2(const DevJob &J, int ilig, int iprt, float pm)
{
  const float *lc = J.lcenter + 3 * GD_AT(ilig, J.nlig, kSiteLigConf);
  const float *pc = J.pcenter + 3 * GD_AT(iprt, J.nprt, kSitePrtConf);
  T dst = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const T t = sub_(add_((T)lc[i], (T)__shfl_sync(0xffffffffu, pm, i)), (T)pc[i]);
    dst = fma_(t, t, dst);
  }
  return dst;
}

// The factor of a hydrogen-bond sum (the FP32 tables carry a factor c, see
// DevParams) and of a KDE sum.
template <int PREC>
__device__ __forceinline__ RealOf<PREC> scaled_sum(int i, RealOf<PREC> x, const DevParams *par)
{
  if constexpr (PREC == kFP64) return i == 6 ? x / (double)par->kde3 : x;
  else return i == 4 ? mul_(x, par->hdb_cinv) : i == 6 ? mul_(x, par->kde3_inv) : x;
}

// Term i (0..8) from its scaled sum x: the value before the per-atom division
// and normalisation (raw), and its normalised form,
// kernel_cuda_l1_montecarlo.cu:460-476.
template <int PREC>
__device__ __forceinline__ RealOf<PREC> raw_term(int i, RealOf<PREC> x, int nmcs)
{
  using T = RealOf<PREC>;
  if (i == 4) return mul_(x, PREC == kFP64 ? (T)kSqrt2PiInvNegD : (T)kSqrt2PiInvNeg);
  if (i == 7) return log(x / (T)nmcs);
  if (i == 8) return sqrt(x);
  return x;
}
template <typename T>
__device__ __forceinline__ T norm_term(int i, T raw, const DevParams *par, int L)
{
  const T v = i < 7 ? raw / (T)L : raw;
  return fma_((T)par->a_para[i], v, (T)par->b_para[i]);
}

}  // namespace gd
