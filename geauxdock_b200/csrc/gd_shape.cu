// gd_shape.cu -- launch shapes of the batched kernel: the warps a replica gets.
#include <algorithm>
#include <cmath>
#include <functional>
#include <queue>
#include <utility>
#include <vector>

#include "gd_pack.h"

namespace gd {

// SMs that no replica's team needs evaluate the steps that may follow
// (gd_spec.cuh): the largest cluster for which one wave holds a cluster per
// replica.  Measured on clusters of 1, 2, 4, 8 and 16: 400 steps of one replica of
// 24 atoms x 600 points on 8 warps' sums 3.41 / 2.34 / 1.65 / 1.27 / 1.01 ms,
// a Dock call of 200 steps 1.65 / 1.16 / 0.85 / 0.67 / 0.61 ms, of 51 replicas x
// 100 steps (34 x 344) 1.01 / 0.79 ms; sizes between lie between (10: 1.17 and
// 0.67 ms).  Two teams of 8 warps in a CTA, for twice the nodes, are slower at
// every size (16 nodes on 8 SMs: 1.52 and 0.81 ms).
static void choose_cluster(const ShapeQuery &q, TileConfig &tc, long long items)
{
  if (q.mode != 0 || tc.group < 8 || tc.warps_per_cta != tc.group) return;
  TileConfig t = tc;
  t.cluster = (int)std::min<long long>(kMaxCluster, q.nsm / std::max(1LL, items));
  for (; t.cluster > 1; --t.cluster)
    if (items <= cluster_occupancy(q.precision, t, q.smem(t))) {
      tc = t;
      return;
    }
}

// CTAs that the registers of the GPU's SMs could hold: a launch with more is not asked about, since the first question
// about a kernel loads its code.
static long long register_wave(const ShapeQuery &q, const TileConfig &tc)
{
  const int regs = q.precision == kFP64 || tc.group >= 8 || tc.wide ? 128 : 80;  // gd_mc.cu, gd_team.cuh
  return 65536LL / (regs * 32 * tc.warps_per_cta) * q.nsm;
}

// A team is the best use of a warp that no replica needs.  Measured per step of
// an ensemble of n replicas (40 atoms x 1500 points) on 1, 2, 4, 8 and 16 warps
// each, where one wave holds the teams: n = 48 128 / 77 / 44 / 22 / 19 us;
// n = 160 129 / 79 / 48 / 33 us; n = 400 130 / 91 / 57 us; n = 880
// 151 / 109 / 84 us; n = 1760 179 / 166 us; and in the same order of G for 24
// atoms x 600 points and 60 x 2000.  The larger team always wins while its wave
// holds, so the line is where the wave ends.
bool choose_team(const ShapeQuery &q, TileConfig &tc, int &grid)
{
  // a team's sums are those of the pair tile 4 x 8 (or of a split order): another tile asked for runs on one warp
  if (tc.split == 1 && q.precision != kFP64 && (tc.kpl != 4 || tc.ab != 8)) return false;
  for (int G = 16; G >= 2; G /= 2)
    for (int R = 1; R * G <= kMaxCtaThreads / 32; ++R) {  // the fewest teams per CTA: they spread over the SMs
      TileConfig t = tc;
      t.group = G;
      t.warps_per_cta = R * G;
      // teams of 8 and 16 read the pocket from shared memory (one CTA per SM whatever it stages)
      t.stage = q.stage_opt > 0 || (q.stage_opt < 0 && G >= 8) ? 1 : 0;
      if (t.stage && q.smem(t) > kSmemLimit) t.stage = 0;
      const size_t smem = q.smem(t);
      if (smem > kSmemLimit) continue;
      const long long items = q.items(R);
      if (items > register_wave(q, t) || items > (long long)kernel_occupancy(q.mode, q.precision, t, smem) * q.nsm) continue;
      tc = t;
      choose_cluster(q, tc, items);
      grid = (int)std::max(1LL, items);
      return true;
    }
  return false;
}

// One warp per replica where one wave holds them all: the replicas per CTA that
// load the fullest SM least, since a step takes about as long as that SM needs
// (2816 replicas of 40 atoms x 1500 points: 32 warps on the fullest SM 281 us a
// step, 20 warps 248 us).
bool choose_spread(const ShapeQuery &q, TileConfig &tc, int &grid)
{
  long long best = -1;
  for (int w = kMaxCtaThreads / 32; w >= 2; --w) {
    TileConfig t = tc;
    t.group = 1;
    t.warps_per_cta = w;
    t.stage = q.stage_opt > 0 ? 1 : 0;
    const size_t smem = q.smem(t);
    if (smem > kSmemLimit) continue;
    const long long items = q.items(w), load = (items + q.nsm - 1) / q.nsm * w;
    if (best >= 0 && load >= best) continue;
    t.wide = load <= 16 && q.precision != kFP64 && t.kpl == 4 && t.ab == 8;
    if (items > register_wave(q, t) || items > (long long)kernel_occupancy(q.mode, q.precision, t, smem) * q.nsm) continue;
    best = load;
    tc = t;
    grid = (int)std::max(1LL, items);
  }
  return best >= 0;
}

// How long a step of the launch takes by a model of it: the work items, heaviest
// first, on `slots` CTAs.  An atom pair against 32 points takes a warp 150 + 62 w
// cycles beside w warps on its scheduler (80 atoms x 2200 points, 8, 9-12, 16 and
// 24 warps per SM: 278, 338, 394 and 606 of them; with 128 registers 120 + 64 w);
// a team of 2 or 4 takes 1.3 times its share of that (8 x 2 warps 465 / 2, 4 x 4
// warps 514 / 4).
static double step_cycles(const ShapeQuery &q, const TileConfig &tc, long long slots)
{
  std::vector<std::pair<double, long long>> load;
  q.loads(tc.warps_per_cta / tc.group, load);
  std::sort(load.begin(), load.end(), [](const auto &a, const auto &b) { return a.first > b.first; });
  long long items = 0;
  for (const auto &l : load) items += l.second;
  slots = std::max(1LL, std::min(slots, items));
  const double w = std::ceil((double)((slots + q.nsm - 1) / q.nsm * tc.warps_per_cta) / 4.0);
  const double alone = tc.wide && tc.group == 1 ? 120.0 + 64.0 * w : 150.0 + 62.0 * w;
  const double per = alone * (tc.group > 1 ? 1.3 : 1.0) / tc.group / 64.0;
  std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
  for (long long i = 0; i < slots; ++i) free_at.push(0.0);
  double last = 0.0;
  for (const auto &l : load)
    for (long long i = 0; i < l.second; ++i) {
      const double t = free_at.top() + l.first * per;
      free_at.pop();
      free_at.push(t);
      last = std::max(last, t);
    }
  return last;
}

// Jobs of uneven sizes: with one warp per replica a step of the whole launch takes
// what the largest replica takes one warp, while the warps of the small ones have
// long finished; teams in several waves, largest first, share it out.  400
// replicas each of 20, 33, 45 and 80 atoms against 2200 points, one wave of one
// warp 493 us a step, 2 or 4 teams of 4 per CTA 333 us; of 8, 14, 25 and 70 atoms
// 431 and 217 us, against 800 points 140 and 106 us; but of 40, 42 and 45 atoms
// 266 and 305 us, of 80 alone 493 and 543 us.  So by the model above, where it
// says an eighth less (teams of 8 and 16 are not: their few half rows per warp
// follow no such rule).  The model's constants are those of the FP32 loop; in FP64 it
// was measured by itself, over eight mixes of ligands x 300, 800 and 2200 points x 4, 8 and
// 12 temperatures (600 to 4200 replicas): where it chooses waves they are 1.1 to 3 times as
// fast as the shape before (20, 45 and 80 atoms x 2200, 1200 replicas, 1500 -> 789 us
// a step; 80 alone, 2400 replicas, 2937 -> 2426), and elsewhere it leaves the shape.
void choose_waves(const ShapeQuery &q, TileConfig &tc, int &grid)
{
  if (q.mode != 0 || !q.loads || tc.group > 4 || (tc.split == 1 && q.precision != kFP64 && (tc.kpl != 4 || tc.ab != 8)))
    return;
  if (q.items(1) > 32LL * q.nsm) return;  // long past one wave even of one warp each
  double best = 0.875 * step_cycles(q, tc, grid);
  const TileConfig base = tc;
  for (const int G : {4, 2})
    for (const int warps : {16, 8}) {
      TileConfig t = base;
      t.group = G;
      t.warps_per_cta = warps;
      t.stage = q.stage_opt > 0 ? 1 : 0;
      if (t.stage && q.smem(t) > kSmemLimit) t.stage = 0;
      const size_t smem = q.smem(t);
      if (smem > kSmemLimit) continue;
      const long long slots = (long long)kernel_occupancy(q.mode, q.precision, t, smem) * q.nsm;
      if (slots < 1) continue;
      const double c = step_cycles(q, t, slots);
      if (c >= best) continue;
      best = c;
      tc = t;
      grid = (int)std::max(1LL, std::min(slots, q.items(warps / G)));
    }
}

}  // namespace gd
