// Segment lengths of the strip march's launches (host logic without CUDA calls).
#pragma once

#include <cmath>

namespace le2d {

// The segment length L that minimises a model of the launch time fitted to measured
// launches,
//   time ~ (w + beta + alpha (ceil(w) - w)) (L + h) (1 + kappa L / 128),   w = tiles / resident tiles,
// w being the launch's waves of tiles, L + h the rows of a tile's march (h for its halo rows
// and the fill of its pipeline), alpha the charge for the idle part of the last wave and
// kappa one for long tiles (the tiles resident at a time then span more rows of the grid).
// L is one of the lengths the fit measured.  Fits:
//   warp-pair (two-step) variants, the FP32 default with its boundary tiles dealt out first,
//   measured on 2048^2 to 16384^2, 8192 x 2048 and 2048 x 8192 with segments of 32 to 256
//   rows: h = 10, beta = 0.1, alpha = 0.5, kappa = 0.02 -- the fastest measured length on
//   each of those grids (an earlier fit without the length term: up to 7 % below it, e.g.
//   147.4 against 158.3 Gnu/s on 3000^2, 155.1 against 158.4 on 4096^2; the earlier rule of
//   about 8 waves of tiles: up to 13 % below it);
//   warp-pair variants launched in halves (le2d_api.cu), w counting the tiles of one half:
//   h = 14, beta = 0, alpha = 0.2, kappa = 0 -- fitted on the same grids with the halves
//   forced on, it picks the fastest measured length, and the halves with it beat the best
//   whole launches on each of those grids but 2048^2 (2 % below): e.g. 4096^2 176.2 against
//   158.5, 8192 x 2048 179.5 against 158.7, 8192^2 195.2 against 181.8 Gnu/s;
//   the FP64 default, variant 15 (one step, 12 warps per SM), measured on 1000^2 to 6000^2,
//   8192 x 2048, 2048 x 8192 and grids of 100 to 250 rows with segments of 8 to 256 rows:
//   h = 8, beta = 0.4, alpha = 0.6, kappa = 0.05 -- within 5 % of the fastest length of at least
//   16 rows on each (multiples of 32 rows: the lengths between them won by 3 % at most and cost the
//   model 20 % where it took them for others); the fit below picked lengths up to 22 % slower, us
//   a step with it / now: 1800^2 84.7 / 74.0, 2048^2 108.2 / 95.3, 16384 x 128 61.7 / 53.2;
//   the other FP64 one-step variants: h = 8, beta = 0.3, alpha = 0, kappa = 0.1, fitted to variant
//   15 while it ran at 16 warps per SM as most of them do, on 2048^2 to 12000^2 and 8192 x 2048
//   (within 1 % of the fastest length on each);
//   FP64 launched in halves, with the waves of one half: h = 8, beta = 0, alpha = 0.2, kappa = 0.1
//   -- the fastest measured length on each of those grids (2-3 % above the whole launches' lengths
//   in halves: 8192^2 58.8 against 57.3, 2048^2 48.1 against 46.5 Gnu/s).
// Where a warp-pair model picks its shortest length, 32 rows, the grid has too few tiles to fill
// the device and its launch lasts as long as one tile's rows march: shorter segments end sooner.
// Two more models choose those, fitted on 1200 x 900 to 3001 x 1777 with segments of 8 to 48
// rows: in halves h = 18, beta = 0.5, alpha = 0 (within 0.5 % of the fastest measured length on
// each), whole h = 6, beta = 0, alpha = 0.5 (the fastest on each).  us a step in halves at 32
// rows / at the length picked: 2048 x 1024 23.7 / 19.1, 1500^2 26.4 / 20.7, 2050 x 1500 27.0 / 24.4,
// 4000 x 1000 30.2 / 27.6, 2048^2 31.0 / 29.9; whole, 2048 x 1024 22.7 / 18.6.
struct SegModel {
  double h, beta, alpha, kappa;
  const int* lens;
  int nlens;
};
constexpr int kPairLens[] = {32, 48, 64, 80, 96, 128, 160, 192, 256};
constexpr int kDefaultLensF64[] = {16, 32, 64, 96, 128};
constexpr int kStepLensF64[] = {16, 24, 32, 40, 48, 56, 64, 80, 96, 112, 128};
constexpr SegModel kPairModel{10.0, 0.1, 0.5, 0.02, kPairLens, 9};
constexpr SegModel kPairHalvesModel{14.0, 0.0, 0.2, 0.0, kPairLens, 9};
constexpr int kShortLens[] = {8, 10, 12, 16, 20, 24, 28, 32};
constexpr SegModel kPairShortModel{6.0, 0.0, 0.5, 0.0, kShortLens, 8};
constexpr SegModel kPairShortHalvesModel{18.0, 0.5, 0.0, 0.0, kShortLens, 8};
constexpr SegModel kDefaultModelF64{8.0, 0.4, 0.6, 0.05, kDefaultLensF64, 5};
constexpr SegModel kStepModelF64{8.0, 0.3, 0.0, 0.1, kStepLensF64, 11};
constexpr int kStepHalvesLensF64[] = {16, 24, 32, 48, 64, 96, 128};
constexpr SegModel kStepHalvesModelF64{8.0, 0.0, 0.2, 0.1, kStepHalvesLensF64, 7};

inline int model_segment(const SegModel& m, int ny, int nstrips, int resident_tiles, int min_len) {
  int best_len = min_len < ny ? min_len : ny;
  double best = 1e300;
  for (int i = 0; i < m.nlens; ++i) {
    if (m.lens[i] < min_len) continue;
    const int l = m.lens[i] < ny ? m.lens[i] : ny;
    const double w = (double)nstrips * ((ny + l - 1) / l) / resident_tiles;
    const double t = (w + m.beta + m.alpha * (std::ceil(w) - w)) * (l + m.h) * (1.0 + m.kappa * l / 128.0);
    if (t < best) {
      best = t;
      best_len = l;
    }
    if (l == ny) break;
  }
  return best_len;
}

}  // namespace le2d
