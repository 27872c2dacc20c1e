// gd_noalloc.cu -- pose energies without any memory allocation.
//
// Who needs this: callers that cannot call cudaMalloc/cudaFree around a
// docking call.  Examples: a host process whose device memory is owned by
// another allocator (a framework's caching allocator or a pool reserved at
// start-up), where a raw cudaMalloc would take memory that allocator has
// already accounted for; and latency-bound serving loops, where cudaFree
// synchronises the whole device and would stall every other stream's docking
// work.  gd_eval_poses() takes host buffers and a device block that it may have
// to allocate; gd_eval_poses_noalloc() does the same work with caller-provided device
// buffers for inputs and outputs, and keeps its own scratch (the packed
// device layout of the Complex, written by the device packer of
// gd_devpack.cu) in one fixed-size array declared below.
//
// The scratch array is a file-scope __device__ variable: every GPU that loads
// libgdock.so holds it (gd_noalloc_scratch_bytes(): 5.60 MiB) until the
// process exits.  Its size covers
// the reference Complex's own capacity (64 ligand atoms, 64 ligand
// conformations, 20 protein conformations of up to 2048 points, 10240 KDE
// points, 512 MCS rows); inputs beyond that are rejected with GD_E_CAPACITY.
// All calls on a device share the array and it keeps the last call's
// contents, so calls whose GPU work overlaps (different streams, or different
// host threads) race on it: issue them one after another.
//
// The poses run in the batched kernels' mode 2 (gd_mc.cu, gd_team.cuh): no work
// items or queue, the pair tables built per CTA, the conformations read through
// L1, and the pocket-specific cells 4 bytes each, which fit where the dense
// potential was.  4096 poses of 40 atoms x 1500 points x 11 conformations in FP32:
// the former kernel, one type group of atoms at a time in scalar arithmetic, 991
// us, now 450 us (bound by the pair loop as the Monte Carlo kernel is); the whole
// call 1.27 -> 0.49 ms.  A pose's FP32 sums are combined in one of two orders, by the
// number of poses sent with it (na_tile, noalloc_shape).
#include <algorithm>
#include <mutex>

#include "gd_pack.h"

namespace gd {
namespace {

constexpr int kNaMaxDevices = 64;

// Layout of the scratch array: the packed job (gd_internal.h) at the largest
// size a reference Complex can describe.
struct NoAllocScratch {
  DevJob job;
  DevParams par;
  int err[4];     // flag, failure kind, field id, value (cleared at the start of every call)
  int2 lgrp[GD_MAXLIG];
  int ncdc[GD_MAX_CONF_PRT];
  float lcenter[GD_MAX_CONF_LIG * 3];
  float pcenter[GD_MAX_CONF_PRT * 3];
  float tcc[GD_MAX_MCS_ROW];
  float4 lig[GD_MAX_CONF_LIG * GD_MAXLIG];
  int4 kslot[2 * GD_MAXKDE];
  float4 mcs[GD_MAXLIG * GD_MAX_MCS_ROW];
  float4 pos[GD_MAX_CONF_PRT * GD_MAXPRO];
  float2 aux[GD_MAX_CONF_PRT * GD_MAXPRO];
  int pcell4[GD_MAX_CONF_PRT * kLigTypes * GD_MAXPRO];
  int pcell_cnt[GD_MAX_CONF_PRT];
  float4 ref4[kLigTypes * kTabCols];
};

}  // namespace

static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoAllocScratch)];

namespace {
std::mutex g_na_mu;
void *g_na_ptr[kNaMaxDevices] = {nullptr};

// Launch shape of n poses: chosen for the caps (the sizes are on the GPU), so it
// depends on the device, the precision and n alone.  The occupancies behind it
// are looked up once per device and precision.
struct NaShapes {
  bool known = false;
  int nsm = 0;
  int wave[5][17] = {};  // [log2 warps per pose][poses per CTA]: CTAs one wave holds
};
NaShapes g_na_shape[kNaMaxDevices][3];

// In FP32 the rows of pass 1 are 64 points, one warp per pose or (the split order
// of 2) a team, and the sums compensated whichever FP32 precision is asked for: rows
// of 128, the other kernels' order, are 7 % faster (4096 poses of 40 x 1500, 461 us a
// call against 495) but their longer chains of plain additions lose more: rms error
// of the raw terms against 64 bits, 40 x 1500, 20 x 400 and 64 x 2048, 1.6, 0.85 and
// 1.3e-7 against 0.88, 0.62 and 0.79e-7 (the former kernel of this call: 1.9, 0.77
// and 0.87e-7).  Over eight sizes from 8 x 200 to 64 x 2048, against that kernel's rms
// error in the same precision (geometric means): FP32 0.75-0.92 times in vdw, ele, pmf,
// hpc and the total on one warp, 0.77-0.96 in teams; FP32_KAHAN 0.77-1.00 on one warp, in
// teams vdw 1.18 and the total 1.04 (the two shares' sums are rounded once more before
// they are added), the others 0.77-1.00; single terms at single sizes up to 1.39 (ele at
// 20 x 400).
TileConfig na_tile(int precision, int lg, int R)
{
  const bool fp64 = precision == kFP64;
  return TileConfig{R << lg, fp64 ? 1 : 2, 8, 0, 1 << lg, fp64 || lg == 0 ? 1 : 2};
}

int noalloc_shape(int dev, int precision, int n, TileConfig &tc, int &n_items, int &grid)
{
  std::lock_guard<std::mutex> lk(g_na_mu);
  NaShapes &s = g_na_shape[dev][precision];
  if (!s.known) {
    GD_CUDA(cudaDeviceGetAttribute(&s.nsm, cudaDevAttrMultiProcessorCount, dev));
    for (int lg = 0; lg < 5; ++lg)
      for (int R = 1; R << lg <= kMaxCtaThreads / 32; ++R) {
        const TileConfig t = na_tile(precision, lg, R);
        const size_t smem = kernel_smem_bytes(0, GD_MAXPRO, GD_MAXLIG, precision, t);
        s.wave[lg][R] = smem > kSmemLimit ? 0 : kernel_occupancy(2, precision, t, smem) * s.nsm;
      }
    s.known = true;
  }
  // as choose_team: the most warps per pose for which one wave holds all, else 8 poses a CTA
  for (int lg = 4; lg >= 1; --lg)
    for (int R = 1; R << lg <= kMaxCtaThreads / 32; ++R)
      if ((n - 1) / R < s.wave[lg][R]) {
        tc = na_tile(precision, lg, R);
        grid = n_items = (n - 1) / R + 1;
        return GD_OK;
      }
  if (s.wave[0][8] < 1) return fail(GD_E_CUDA, "the pose kernel cannot launch");
  tc = na_tile(precision, 0, 8);
  n_items = (n - 1) / 8 + 1;
  grid = std::min(n_items, s.wave[0][8]);
  return GD_OK;
}

// The device packer's destination: the scratch array's members.
PackDst scratch_dst(NoAllocScratch *S)
{
  PackDst D{};
  D.job = &S->job;
  D.par = &S->par;
  D.ref4 = S->ref4;
  D.err = S->err;
  D.lgrp = S->lgrp;
  D.lcenter = S->lcenter;
  D.pcenter = S->pcenter;
  D.tcc = S->tcc;
  D.lig = S->lig;
  D.kslot = S->kslot;
  D.mcs = S->mcs;
  D.pos = S->pos;
  D.aux = S->aux;
  D.ncdc = S->ncdc;
  D.pcell4 = S->pcell4;
  D.pcell_cnt = S->pcell_cnt;
  D.pcell_stride = kLigTypes * GD_MAXPRO;
  D.kde_cap = GD_MAXKDE;
  D.Ppad = 0;
  D.nkde_expect = -1;
  D.expect_L = D.expect_nlig = D.expect_nprt = D.expect_M = D.expect_ntmp = -1;
  D.rep = nullptr;
  return D;
}

}  // namespace
}  // namespace gd

using namespace gd;

// Set-up on the calling thread's current device: the device address of the
// scratch array, looked up once per device.  The first call on a device does
// this look-up; make that first call before any stream capture.
static int noalloc_scratch(NoAllocScratch **out)
{
  int dev = 0;
  GD_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNaMaxDevices) return fail(GD_E_INVALID, "device ordinal %d", dev);
  std::lock_guard<std::mutex> lk(g_na_mu);
  if (!g_na_ptr[dev]) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr)
      return fail(GD_E_CUDA, "cudaGetSymbolAddress(scratch) on device %d: %s", dev, cudaGetErrorString(e));
    g_na_ptr[dev] = p;
  }
  *out = (NoAllocScratch *)g_na_ptr[dev];
  return GD_OK;
}

extern "C" size_t gd_noalloc_scratch_bytes(void) { return sizeof(NoAllocScratch); }

extern "C" int gd_eval_poses_noalloc(const Complex *d_complex, int n, const int *d_conf, const float *d_mm,
                                     int precision, float *d_out, float *d_raw, void *stream)
{
  if (!d_complex || n < 0 || (n > 0 && (!d_conf || !d_mm || !d_out))) return fail(GD_E_INVALID, "null argument");
  if (precision < GD_PREC_FP32 || precision > GD_PREC_FP64) return fail(GD_E_INVALID, "precision = %d", precision);
  cudaStream_t st = (cudaStream_t)stream;
  int dev = 0;
  GD_CUDA(cudaGetDevice(&dev));
  if (st != nullptr) {
    // the scratch address below is the current device's: the stream must belong to it
    int sdev = -1;
    GD_CUDA(cudaStreamGetDevice(st, &sdev));
    if (sdev != dev)
      return fail(GD_E_INVALID, "gd_eval_poses_noalloc: the stream belongs to device %d, the current device is %d",
                  sdev, dev);
  }
  NoAllocScratch *S = nullptr;
  GD_TRY(noalloc_scratch(&S));
  if (precision == GD_PREC_FP32) precision = GD_PREC_FP32_KAHAN;  // na_tile
  TileConfig tc = na_tile(precision, 0, 8);
  KArgs a{};
  int grid = 0;
  if (n > 0) GD_TRY(noalloc_shape(dev, precision, n, tc, a.n_items, grid));
  // the failure flag and its details must start at zero on every call
  GD_CUDA(cudaMemsetAsync(S->err, 0, sizeof(S->err), st));
  GD_CUDA(device_pack(d_complex, scratch_dst(S), st));
  if (n > 0) {
    a.jobs = &S->job;
    a.err = &S->err[0];
    a.Pall = GD_MAXPRO;
    a.lig_slots = GD_MAXLIG;
    a.n_poses = n;
    a.conf = d_conf;
    a.mm = d_mm;
    a.out = d_out;
    a.raw = d_raw;
    GD_CUDA(launch_kernel(2, precision, tc, a, grid, st));
  }
  int h[4] = {0, 0, 0, 0};
  GD_CUDA(cudaMemcpyAsync(h, S->err, sizeof(h), cudaMemcpyDeviceToHost, st));
  GD_CUDA(cudaStreamSynchronize(st));
  if (h[0] & kErrPack) {
    if (h[1] == kPackFailCapacity)
      return fail(GD_E_CAPACITY, "gd_eval_poses_noalloc: %s = %d exceeds the fixed scratch (%zu B, sized for the "
                                 "reference Complex caps)", pack_field_name(h[2]), h[3], sizeof(NoAllocScratch));
    return fail(GD_E_INVALID, "gd_eval_poses_noalloc: invalid %s: %d", pack_field_name(h[2]), h[3]);
  }
  if (h[0]) return fail(GD_E_INVALID, "gd_eval_poses_noalloc: a pose's conformation index is out of range");
  return GD_OK;
}
