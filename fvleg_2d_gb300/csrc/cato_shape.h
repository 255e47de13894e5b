// cato_shape.h -- the launch shapes of the stage kernels as functions of the grid: the rules only, so
// that a host test can read them without CUDA.
#pragma once

#include <algorithm>
#include <vector>

#include "../../include/cato_gpu.h"

namespace cato {

// The shape of a single-grid launch: CTA columns incl. the x-halo, rows marched per CTA, and for
// the edge-parallel kernels (FP64, double-float) the rows of a block and the register budget.
struct StageShape {
  int width = 128;  // the plan's CTA width, as the caller knows it
  int threads = 128;
  int rows = 64;
  int block = 4;
  int warps = 9;    // blockDim.y of the edge-parallel kernels, at least 2 block + 1
  int variant = 0;
};

// The kernel of a shape: the FP64 register budget (the other types have one kernel, whatever budget
// was set) and the split form, which FP64 has at the default budget only.
struct StageForm {
  int variant;
  bool split;
};
inline StageForm stage_form(const StageShape& s, int precision) {
  const int variant = precision == CATO_FP64 ? s.variant : 0;
  return {variant, precision != CATO_MIXED && variant == 0 && s.warps > 2 * s.block + 1};
}

// tiles of columns (incl. the halo) x rows
inline long long tiles_of(int ni, int nj, int ng, int columns, int rows) {
  const int W = columns - 2 * ng;
  return (long long)((ni + W - 1) / W) * ((nj + rows - 1) / rows);
}

// The shape of a plan (CTA width incl. the halo, rows per CTA), as cato_gpu_set_plan takes it and
// cato_gpu_get_plan gives it; every shape is one of these.  The edge-parallel kernels take half the
// width in columns (32 .. 128) and march in blocks of up to 4 rows.
inline StageShape plan_shape(int sms, int ni, int nj, int ng, int precision, int width, int rows) {
  StageShape s;
  s.rows = rows;
  s.width = s.threads = width;
  if (precision == CATO_MIXED) return s;
  s.threads = width / 64 * 32;
  s.block = std::min(rows, s.threads > 64 ? 2 : 4);
  s.warps = 2 * s.block + 1;
  // the split form, where a CTA is a single block of 1 or 2 rows and SMs stay idle
  if (s.threads == 32 && rows == 1 && tiles_of(ni, nj, ng, 32, 1) <= sms) s.warps = 12;
  if (s.threads == 32 && rows == 2 && tiles_of(ni, nj, ng, 32, 2) <= 2 * sms + 16) s.warps = 10;
  return s;
}

// Default single-grid launch shape, for a GPU of sms SMs (measured on 152).
//
// FP32 strips of 64 columns: as many rows per CTA (32 .. 1) as leave the GPU about full; a strip
// of r rows pays for r + 1.5 of them, and more than 32 leave a long last wave (3000 x 2010 Roe:
// 772 us a step at 32 rows, 1022 at 64 rows of 128 columns; 4096^2 HLLC 1257 and 1279). Best of 1
// .. 64 rows: 64 x 48 and 200^2: 1 row, 300^2: 1 or 2 (24.6 and 25.9 us, 32.5 at 4), 512^2: 4,
// 1024^2: 16.
//
// Edge-parallel tiles (FP64, double-float).  While they leave SMs idle the chain of a block is the
// time of the launch: 32 columns in the split form with a single block of 1 row (64 x 48 HLLC:
// 40 us a step, 54 in the unsplit form) or 2 rows (128 x 100: 59 us, 62 unsplit at 4 rows; a little
// beyond two tiles per SM too, where 4 rows give a few SMs a second tile: 392 x 44 to 448 x 40, 308
// to 320 tiles, HLLC 70 to 72 us, 77 to 79 at 4 rows, double-float 37 and 35), then a single
// unsplit block of 4 (200^2: 116 us, 149 with 64 columns).  From two tiles per SM on 64
// columns, blocks of 4 rows and as many blocks per CTA as leave about four waves of the two resident
// CTAs (1024^2: 1735 us at 8 rows, 1790 at 32; 4096^2: 24.0 ms at 32 rows, 25.3 at 8).  With two ghost
// columns a side a little later (256^2: 170 us, 191 with 64 columns; Roe 239 and 251, double-float 69
// and 78); with three, 32 columns lose more to the halo (SLAU + MLP5 357 and 344).
inline StageShape default_shape(int sms, int ni, int nj, int ng, int precision) {
  auto tiles = [&](int columns, int rows) { return tiles_of(ni, nj, ng, columns, rows); };
  auto plan = [&](int width, int rows) {
    return plan_shape(sms, ni, nj, ng, precision, width, rows);
  };
  // a launch has at most 65535 tiles along j: taller grids (2 M rows at 32) take taller tiles
  auto fit = [&](int rows) {
    while ((nj + rows - 1) / rows > 65535) rows *= 2;
    return rows;
  };
  if (precision == CATO_MIXED) {
    int rows = 32;
    while (rows > 2 && tiles(64, rows) < 7LL * sms) rows /= 2;
    if (tiles(64, 2) < 3LL * sms) rows = 1;  // 200^2: 20.4 us a step, 23.0 at 2 rows
    return plan(64, fit(rows));
  }
  for (int rows : {1, 2}) {
    const StageShape s = plan(64, rows);
    if (s.warps > 2 * s.block + 1) return s;
  }
  if (tiles(64, 4) < (ng == 2 ? 7LL * sms / 3 : 2LL * sms)) return plan(64, 4);
  int rows = 32;
  while (rows > 4 && tiles(64, rows) < 7LL * sms) rows /= 2;
  return plan(128, fit(rows));
}

// The candidates of a tuning run: the current plan and the widest one, each with the current, half
// and a quarter of the rows per CTA (down to 8), and with every FP64 register budget; none wider
// than the grid with its halo.
inline std::vector<StageShape> tune_shapes(int sms, int ni, int nj, int ng, int precision,
                                           const StageShape& current) {
  std::vector<StageShape> out;
  const int r = current.rows;
  const int half_rows = r <= 8 ? r : std::max(8, r / 2);
  const int quarter_rows = r <= 8 ? r : std::max(8, r / 4);
  const int nvar = precision == CATO_FP64 ? 3 : 1;
  for (int v = 0; v < nvar; ++v) {
    for (int width : {current.width, 256}) {
      for (int rows : {r, half_rows, quarter_rows}) {
        StageShape q = plan_shape(sms, ni, nj, ng, precision, width, rows);
        q.variant = v;
        bool dup = false;
        for (const StageShape& x : out)
          dup |= x.width == q.width && x.rows == q.rows && x.variant == q.variant;
        // (the current plan by its columns: a width of 128 is 64 columns in FP64)
        const int span = width == current.width ? q.threads : width;
        if (!dup && span - 2 * ng <= ni + 2 * ng) out.push_back(q);
      }
    }
  }
  return out;
}

// Rows per tile of a batch, at most the plan's, for grids of ni x nj cells in strips of W columns.
// FP32 strips hide their latency with neighbours: the most rows that leave five tiles per SM (served
// stream, 1.1 M cells: 1.93 ms per 16 steps at 8 rows, 3.06 at 32).  The edge-parallel tiles fill an
// SM with two: what counts is the share of the busiest SM, its tiles times their rows and 1.2 more
// for what a tile repeats, its ghost rows and lowest edges (one wave of 304 tiles of 4 to 32 rows
// takes k (r + c), c = 0.8 for FP64 HLLC and Roe, 1.1 with MLP5, 1.6 for double-float; 16 steps of
// an FP64 sweep of 0.29 M cells: 19.9 ms at 4 rows with 9 tiles on an SM, 24.4 at 16 rows with 3;
// MLP5, 16 grids up to 512^2: 21.7 ms at 24 rows with 2, 25.0 at 16 with 3), over the multiples of
// four up to the tallest grid.
struct BatchGrid {
  int ni, nj, W;
};
inline int batch_rows(int sms, int precision, int plan_rows, const std::vector<BatchGrid>& grids) {
  auto n_tiles = [&](int r) {
    long long n = 0;
    for (const BatchGrid& g : grids) {
      const int rr = std::min(r, g.nj);
      n += (long long)((g.ni + g.W - 1) / g.W) * ((g.nj + rr - 1) / rr);
    }
    return n;
  };
  int rows = plan_rows;
  if (precision == CATO_MIXED) {
    while (rows > 4 && n_tiles(rows) < 5LL * sms) rows = std::max(4, rows / 2);
    return rows;
  }
  auto share = [&](int r) { return (double)((n_tiles(r) + sms - 1) / sms) * (r + 1.2); };
  int tallest = 1;
  for (const BatchGrid& g : grids) tallest = std::max(tallest, g.nj);
  rows = std::min(rows, (int)(((long long)tallest + 3) / 4 * 4));
  double least = share(rows);
  for (int r = (rows - 1) / 4 * 4; r >= 4; r -= 4) {
    const double x = share(r);
    if (x < least) {
      least = x;
      rows = r;
    }
  }
  return rows;
}

}  // namespace cato
