// wf_price.h -- which form of the step an automatic grid runs: the cheapest by
// what each form costs on a B200, computed from what its kernels launch.
//
// The prices are linear in those counts, in microseconds a step.  Their
// coefficients are non-negative least squares over 1274 grids timed in every
// form (16 x 24 x 24 to 1024^3 cells, x extents that leave a brick or a tile
// partly outside, 0- to 48-cell CPML on any axes, zero and periodic boundaries,
// exact and FMA, FP32 and 16-bit; fields of noise).  Over those grids the form
// picked takes 0.2 % more than the best one on average (0.2 % too on a half left
// out of the fit), 10 of them more than 6 %.  A rule on the cells alone lost up
// to 1.8x: bricks cost the same with 8 of their 32 columns inside as with all
// (16 x 256 x 256, periodic: split 24 us, bricks 44), and the interior of a mixed
// step pays for whole 128-cell tiles.
//
// Host code without CUDA types: compiles on its own.
#pragma once
#include <algorithm>
#include <cmath>

namespace wf {

// A grid as the rule sees it: cells, CPML depth at each end (0: none).
struct StepShape {
  int n[3];
  int depth[3];
  bool periodic[3];
  bool b16;  // 16-bit storage
};

enum class StepForm { kSplit, kMarch, kBrick, kMix };

// Where bricks and marching tiles can share a step: the marching tiles'
// interior, cells whose step, halo and warm-up plane meet no slab.
struct InteriorBox {
  int lo[3], hi[3];
};

namespace price {

constexpr int kBrick[3] = {32, 8, 4};
constexpr int kTileWide = 128, kTileRows = 4, kColumnWide = 16, kColumnRows = 32;
constexpr double kSms = 148.0;
constexpr double kMarchSlots = 3 * kSms;  // marching CTAs resident at once
constexpr double kWarmup = 1.5;           // planes a marching item pays before its first

inline int pieces(int n, int size) { return (n + size - 1) / size; }

// Of the pieces of `size` cells along an axis of n cells, those whose cells or
// whose halo below meet the CPML slabs of depth t.
inline int meeting(int n, int size, int t) {
  if (t <= 0) return 0;
  const int all = pieces(n, size), low = std::min(t / size + 1, all);
  const int high = std::max(low, std::min(all, std::max(0, n - t) / size));
  return low + all - high;
}

inline bool has_cpml(const StepShape &s) { return s.depth[0] | s.depth[1] | s.depth[2]; }
inline bool any_periodic(const StepShape &s) { return s.periodic[0] || s.periodic[1] || s.periodic[2]; }
inline double mcells(const int n[3]) { return 1e-6 * n[0] * n[1] * static_cast<double>(n[2]); }

// Cells in the slabs of an axis, in millions.
inline double slab_mcells(const StepShape &s, int a) {
  return mcells(s.n) * std::min(2 * s.depth[a], s.n[a]) / s.n[a];
}

// Bricks of the grid, the same in thousands, and the thousands that meet each
// axis's slabs (counted once per axis).
struct BrickCounts {
  double count, all, meet[3];
};
inline BrickCounts bricks(const StepShape &s) {
  double t[3], m[3];
  for (int a = 0; a < 3; ++a) {
    t[a] = pieces(s.n[a], kBrick[a]);
    m[a] = meeting(s.n[a], kBrick[a], s.depth[a]);
  }
  return BrickCounts{t[0] * t[1] * t[2],
                     1e-3 * t[0] * t[1] * t[2],
                     {1e-3 * m[0] * t[1] * t[2], 1e-3 * m[1] * t[0] * t[2], 1e-3 * m[2] * t[0] * t[1]}};
}

// z chunk of the marching tiles over a box of m cells: 24 planes (fewer
// warm-up planes) while they still give four waves of items, else 12; 16-bit
// storage, whose kernel is issue-bound, 32, or 48 from 1024 planes on.
inline int march_chunk(const int m[3], int nz, bool b16) {
  if (b16) return nz >= 1024 ? 48 : 32;
  const double items = static_cast<double>(pieces(m[0], kTileWide)) * pieces(m[1], kTileRows) * pieces(m[2], 24);
  return items >= 4 * kMarchSlots ? 24 : 12;
}

// One launch of bricks (wf_brick_impl.cuh): every brick alike, whatever part
// of it is inside; CPML code per axis that a brick meets, dearer on x where the
// slabs split groups of four; waves of 2 (with CPML) or 3 CTAs an SM; the
// wrapped cells of periodic axes.
inline double brick_us(const StepShape &s) {
  const BrickCounts k = bricks(s);
  const bool pml = has_cpml(s), odd = s.depth[0] % 4 != 0;
  const double cells = mcells(s.n), slots = (pml ? 2 : 3) * kSms;
  const double waves = 1e-3 * slots * std::ceil(k.count / slots);
  if (s.b16) {
    if (!pml) return 4.13 + 0.721 * k.all + 0.6 * cells + 7.33 * waves;
    return 4.62 + 2.5 * cells + 9.91 * waves + (odd ? 12.3 : 4.59) * k.meet[0] +
           5.38 * (k.meet[1] + k.meet[2]) + 0.378 * odd;
  }
  const bool per = any_periodic(s);
  const double narrow = s.n[0] < kBrick[0] ? k.all : 0.0;  // rows shorter than a brick
  const double xwrap = s.periodic[0] ? 2e-3 * pieces(s.n[1], kBrick[1]) * pieces(s.n[2], kBrick[2]) : 0.0;
  const double both = s.periodic[0] && s.n[0] <= kBrick[0] ? k.all : 0.0;  // x wraps on both sides of a brick
  if (!pml)
    return 1.75 + 8.73 * k.all + 1.71 * waves + 0.562 * narrow + 2.22 * xwrap +
           (per ? 1.76 + 0.772 * k.all : 0.0);
  return 1.14 + 1.76 * k.all + 0.858 * cells + 10.4 * waves + (odd ? 7.01 : 3.73) * k.meet[0] +
         4.15 * (k.meet[1] + k.meet[2]) + 1.36 * odd + 0.953 * narrow + 1.22 * xwrap + 2.19 * both +
         (per ? 1.06 + 1.68 * k.all : 0.0);
}

// The marching tiles (wf_fused_impl.cuh): items of a class of CPML axes, the x
// slabs as column tiles where they are at most 16 cells deep, each item a chain
// of its chunk's planes.
inline double march_us(const StepShape &s) {
  const bool pml = has_cpml(s), odd = s.depth[0] % 4 != 0;
  const bool columns = s.depth[0] > 0 && s.depth[0] <= kColumnWide && s.n[0] >= 3 * kColumnWide;
  const int wide = columns ? s.n[0] - 2 * kColumnWide : s.n[0], chunk = march_chunk(s.n, s.n[2], s.b16);
  const double cells = mcells(s.n), chain = std::min(chunk, s.n[2]) + kWarmup, u = chain / kMarchSlots;
  const double tx = pieces(wide, kTileWide), ty = pieces(s.n[1], kTileRows), tz = pieces(s.n[2], chunk);
  if (!pml) {
    const double items = tx * ty * tz, waves = std::ceil(items / kMarchSlots) * chain;
    if (s.b16) return 30.6 + 0.972 * items * u + 2.06 * std::max(0.0, cells - 4.0);
    return 3.94 + (0.466 + 0.362 * wide / (kTileWide * tx)) * waves + 0.707 * items * u +
           0.476 * std::max(0.0, cells - 4.0);
  }
  const double mx = columns ? 0 : meeting(s.n[0], kTileWide, s.depth[0]);
  const double my = meeting(s.n[1], kTileRows, s.depth[1]), mz = meeting(s.n[2], chunk, s.depth[2]);
  auto items = [&](bool x, bool y, bool z) {  // whose CPML axes are these
    return (x ? mx : tx - mx) * (y ? my : ty - my) * (z ? mz : tz - mz);
  };
  const double cy = columns ? pieces(s.n[1], kColumnRows) : 0, cm = columns ? meeting(s.n[1], kColumnRows, s.depth[1]) : 0;
  auto cols = [&](bool y, bool z) { return 2 * (y ? cm : cy - cm) * (z ? mz : tz - mz); };
  const double xyz = items(true, true, true), cxyz = cols(true, true);
  const double slab_x = slab_mcells(s, 0), slab_yz = slab_mcells(s, 1) + slab_mcells(s, 2);
  const double odd_wide = odd ? mx * ty * tz : 0.0, odd_cols = odd ? 2 * cy * tz : 0.0;
  // more axes cost more an item, split groups on x a surcharge, psi by the cell;
  // the slowest class's chain is there whatever the others take
  if (s.b16)
    return 42.9 +
           u * (1.08 * items(false, false, false) + 0.856 * items(false, true, false) +
                0.994 * items(false, false, true) + 9.83 * items(false, true, true) +
                1.13 * items(true, false, false) + 4.36 * (items(true, true, false) + items(true, false, true)) +
                0.409 * cols(false, false) + 10.8 * (cols(true, false) + cols(false, true)) + 54.9 * cxyz +
                2.42 * odd_wide + 1.26 * odd_cols) +
           1.85 * cells + 23.9 * slab_x + 3.95 * slab_yz + chain * (1.01 * (xyz > 0) + 0.913 * (cxyz > 0));
  return 12.4 +
         u * (0.779 * items(false, false, false) + 0.006 * items(false, false, true) +
              2.12 * items(false, true, true) + 1.41 * items(true, false, false) +
              1.37 * (items(true, true, false) + items(true, false, true)) + 3.35 * xyz +
              3.36 * cols(false, false) + 6.04 * (cols(true, false) + cols(false, true)) + 52.7 * cxyz +
              2.44 * odd_wide + 0.879 * odd_cols) +
         4.4 * cells + 8.02 * slab_x + 13.6 * slab_yz + chain * (1.31 * (xyz > 0) + 2.86 * (cxyz > 0));
}

// Marching tiles over the box and bricks around it, one after the other (the
// marching CTAs leave no room for a brick), a join and a separate tail.
inline double mix_us(const StepShape &s, const InteriorBox &b) {
  const int m[3] = {b.hi[0] - b.lo[0], b.hi[1] - b.lo[1], b.hi[2] - b.lo[2]};
  const int chunk = march_chunk(m, s.n[2], s.b16);
  const double planes = static_cast<double>(pieces(m[0], kTileWide)) * pieces(m[1], kTileRows) * pieces(m[2], chunk) *
                        (std::min(chunk, m[2]) + kWarmup) / kMarchSlots;
  const BrickCounts k = bricks(s);
  const double inner = 1e-3 * (m[0] / kBrick[0]) * (m[1] / kBrick[1]) * (m[2] / kBrick[2]);
  const bool odd = s.depth[0] % 4 != 0;
  const double slabs = slab_mcells(s, 0) + slab_mcells(s, 1) + slab_mcells(s, 2);
  if (s.b16)
    return 17.5 + 1.13 * planes + 1.13 * mcells(m) + 18.1 * (k.all - inner) + (odd ? 7.59 : 1.03) * k.meet[0] +
           1.29 * slabs;
  return 5.61 + 0.578 * planes + 5.32 * mcells(m) + 18.8 * (k.all - inner) + (odd ? 6.33 : 3.03) * k.meet[0] +
         2.0 * slabs;
}

// The H and E pair (wf_split.cu), FP32: 15 us per million cells while the two
// states fit L2 (about 2.5 million cells), 24 beyond; a warp of 32 cells pays
// for the x slab if any of its cells is in it.
inline double split_us(const StepShape &s) {
  const double c = mcells(s.n), out = std::max(0.0, c - 1.0), far = std::max(0.0, c - 2.0);
  if (!has_cpml(s)) return 6.27 + 15.5 * c + 1.88 * out + 6.54 * far;
  const double slab = slab_mcells(s, 0) + slab_mcells(s, 1) + slab_mcells(s, 2);
  const double xwarps = c * meeting(s.n[0], 32, s.depth[0]) / pieces(s.n[0], 32);
  return 7.02 + 15.4 * c + 7.88 * out + 1.88 * far + 2.54 * xwarps + 5.96 * slab;
}

// A batch's step as one launch of every grid's bricks (the CPML instantiation,
// whatever a brick meets) ...
inline double batch_brick_us(const StepShape *grids, int n) {
  double us = 6.32;
  for (int i = 0; i < n; ++i) {
    const StepShape &s = grids[i];
    const BrickCounts k = bricks(s);
    us += 12.5 * k.all + (s.depth[0] % 4 ? 6.24 : 3.09) * k.meet[0] + 6.3 * (k.meet[1] + k.meet[2]) +
          1.51 * mcells(s.n);
  }
  return us;
}

// ... and as one persistent launch of 4-row, 16-plane marching items per CPML
// class that some grid has.
constexpr int kBatchChunk = 16;
inline double batch_march_us(const StepShape *grids, int n) {
  double us = 11.4;
  bool used[8] = {};
  for (int i = 0; i < n; ++i) {
    const StepShape &s = grids[i];
    const double u = (std::min(kBatchChunk, s.n[2]) + kWarmup) / kMarchSlots;
    const int size[3] = {kTileWide, kTileRows, kBatchChunk};
    double all[3], met[3], items[8];
    for (int a = 0; a < 3; ++a) {
      all[a] = pieces(s.n[a], size[a]);
      met[a] = meeting(s.n[a], size[a], s.depth[a]);
    }
    for (int c = 0; c < 8; ++c) {
      items[c] = 1.0;
      for (int a = 0; a < 3; ++a) items[c] *= c >> a & 1 ? met[a] : all[a] - met[a];
      used[c] = used[c] || items[c] > 0.0;
    }
    us += u * (1.03 * items[0] + 2.62 * (items[2] + items[4]) + 14.2 * items[6] + 1.63 * items[1] +
               3.94 * (items[3] + items[5]) + 5.22 * items[7] +
               (s.depth[0] % 4 ? 1.57 * met[0] * all[1] * all[2] : 0.0)) +
          3.31 * mcells(s.n);
  }
  for (bool c : used) us += 6.06 * c;
  return us + 5.97 * used[7];
}

}  // namespace price

// The interior box of a mixed step, cut to whole bricks; false where CPML on x
// or room for a box is missing.
inline bool interior_box(const StepShape &s, InteriorBox *m) {
  for (int a = 0; a < 3; ++a) {
    const int n = s.n[a], t = s.depth[a], b = price::kBrick[a];
    m->lo[a] = t > 0 ? t / b * b + b : 0;
    m->hi[a] = t > 0 ? (n - t) / b * b : n;
    if (m->hi[a] <= m->lo[a]) return false;
  }
  return s.depth[0] > 0;
}

// The cheapest of the forms that can run.  Some prices carry a margin.
// Without CPML a tie goes to the marching tiles (5 % on FP32 bricks, 10 % on
// 16-bit ones), which run up to 7 % faster in memory no grid used before
// (264 x 440 x 320: 352 and 374 us); with periodic axes to the split pair (3 %).
// The split pair is charged 12 % where marching tiles could run: its fit is
// that far off on short rows with slabs, and bricks lose little there.  With
// CPML on x alone marching tiles are charged 5 %: their fit is up to 9 % low on
// 16-cell slabs there (512^3: 1408 us, bricks around them 1368).  The mixed step
// has to be 3.5 % below bricks: its work lists, streams and graphs with forks cost
// a new grid more (256^3 with 8 cells, its first 50 steps: 14.3 ms, bricks 11.9).
inline StepForm cheapest_step(const StepShape &s, bool march_ok, bool brick_ok, bool split_ok) {
  const bool pml = price::has_cpml(s), x_alone = s.depth[0] > 0 && !(s.depth[1] | s.depth[2]);
  StepForm best = StepForm::kSplit;
  double us = 1e300;
  auto offer = [&](StepForm f, double p) {
    if (p < us) {
      us = p;
      best = f;
    }
  };
  InteriorBox box;
  if (march_ok) offer(StepForm::kMarch, price::march_us(s) * (x_alone ? 1.05 : 1.0));
  if (split_ok && !s.b16) offer(StepForm::kSplit, price::split_us(s) * (march_ok ? 1.12 : 1.0));
  if (!brick_ok) return best;
  const double bricks = price::brick_us(s);
  offer(StepForm::kBrick, bricks * (pml ? 1.0 : (s.b16 ? 1.10 : (price::any_periodic(s) ? 1.03 : 1.05))));
  if (march_ok && interior_box(s, &box)) {
    const double mix = price::mix_us(s, box);
    if (mix * 1.035 < bricks) offer(StepForm::kMix, mix);
  }
  return best;
}

// Whether a batch runs as bricks rather than marching items.  Fitted to 142
// batches of 1 to 60 grids timed both ways; the pick is 0.2 % over the better
// one on average.  Bricks always cost 4 % (16 cubes of 128 cells without CPML:
// 460 us against 302; 3 of 512 x 256 x 128 with 8 cells: 770 against 682),
// marching always 72 % (48 cubes of 32 with 10 cells: 270 against 67).  Without
// CPML a tie goes to the marching items, as for one grid.
inline bool batch_takes_bricks(const StepShape *grids, int n) {
  bool pml = false;
  for (int i = 0; i < n; ++i) pml = pml || price::has_cpml(grids[i]);
  return price::batch_brick_us(grids, n) * (pml ? 1.0 : 1.05) < price::batch_march_us(grids, n);
}

}  // namespace wf
