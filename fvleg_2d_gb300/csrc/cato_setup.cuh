// cato_setup.cuh -- host-side derivations shared by every entry point that turns a cato_config
// into kernel arguments (handles, batch slots and the allocation-free residual), so that all of
// them feed the stage kernel the same constants and launch shape for the same configuration.
#pragma once

#include "../../include/cato_gpu.h"
#include "cato_launch.cuh"
#include "cato_physics.cuh"

namespace cato {

// The scheme constants of a configuration (gamma-derived ratios, AUSM+-up coefficients, the
// low-Mach and entropy-fix switches), in FP64; other compute types take convert_consts of it.
inline FluxConsts<double> flux_consts_of(const cato_config& c) {
  const double g = c.gamma;
  FluxConsts<double> K{};
  K.gamma = g;
  K.g_over_gm1 = g / (g - 1.0);
  K.gm1 = g - 1.0;
  K.two_gm1_over_gp1 = 2.0 * ((g - 1.0) / (g + 1.0));
  K.gamma_factor = ((2.0 * (g - 1.0)) / (g + 1.0));
  K.hllc_gf = (g + 1.0) / (2.0 * g);
  K.harten_delta = c.harten_delta;
  K.ausm_beta = c.ausm_beta;
  K.ausm_kp = c.ausm_kp;
  K.ausm_ku = c.ausm_ku;
  K.ausm_sigma = c.ausm_sigma;
  K.cfl = c.cfl;
  K.rdx = 1.0 / c.dx;
  K.rdy = 1.0 / c.dy;
  K.low_mach_fix = c.apply_low_mach_fix ? 1 : 0;
  K.gm1_y62 = intdiv::recip62(intdiv::bits_of(K.gm1));
  K.harten = c.roe_entropy_fix == CATO_ROE_HARTEN ? 1 : 0;
  return K;
}

// Default single-grid launch shape.
//
// FP32 strips of 64 columns: as many rows per CTA (32 .. 1) as leave the GPU about full; a strip
// of r rows pays for r + 1.5 of them, and more than 32 leave a long last wave (3000 x 2010 Roe:
// 772 us a step at 32 rows, 1022 at 64 rows of 128 columns; 4096^2 HLLC 1257 and 1279). Best of 1
// .. 64 rows: 64 x 48 and 200^2: 1 row, 300^2: 1 or 2 (24.6 and 25.9 us, 32.5 at 4), 512^2: 4,
// 1024^2: 16.
//
// Edge-parallel tiles (FP64, double-float).  While they leave SMs idle the chain of a block is the
// time of the launch: 32 columns in the split form with a single block of 1 row (64 x 48 HLLC:
// 40 us a step, 54 in the unsplit form) or 2 rows (128 x 100: 59 us, 62 unsplit at 4 rows), then a
// single unsplit block of 4 (200^2: 116 us, 149 with 64 columns).  From two tiles per SM on 64
// columns, blocks of 4 rows and as many blocks per CTA as leave about four waves of the two resident
// CTAs (1024^2: 1735 us at 8 rows, 1790 at 32; 4096^2: 24.0 ms at 32 rows, 25.3 at 8).  With two ghost
// columns a side a little later (256^2: 170 us, 191 with 64 columns; Roe 239 and 251, double-float 69
// and 78); with three, 32 columns lose more to the halo (SLAU + MLP5 357 and 344).
constexpr int kSMs = 152;
inline StageShape default_shape(int ni, int nj, int ng, int precision) {
  auto tiles = [&](int columns, int rows) {
    const int W = columns - 2 * ng;
    return (long long)((ni + W - 1) / W) * ((nj + rows - 1) / rows);
  };
  StageShape s;
  if (precision == CATO_MIXED) {
    s.threads = 64;
    s.rows = 32;
    while (s.rows > 2 && tiles(64, s.rows) < 7LL * kSMs) s.rows /= 2;
    if (tiles(64, 2) < 3LL * kSMs) s.rows = 1;  // 200^2: 20.4 us a step, 23.0 at 2 rows
    s.width = s.threads;
    return s;
  }
  s.width = 64;
  s.threads = 32;
  if (tiles(32, 1) <= kSMs) {
    s.rows = s.block = 1;
    s.warps = 12;
    return s;
  }
  if (tiles(32, 2) <= 2 * kSMs + 16) {
    s.rows = s.block = 2;
    s.warps = 10;
    return s;
  }
  s.warps = 9;
  s.rows = s.block = 4;
  if (tiles(64, 4) < (ng == 2 ? 7LL * kSMs / 3 : 2LL * kSMs)) return s;
  s.width = 128;
  s.threads = 64;
  s.block = 4;
  s.rows = 32;
  while (s.rows > 4 && tiles(64, s.rows) < 7LL * kSMs) s.rows /= 2;
  return s;
}

// reconstruction kind of a limiter id: 0 = TVD2, 3 = MLP3, 5 = MLP5
inline int recon_of_limiter(int limiter) {
  return limiter == CATO_LIM_MLP3 ? 3 : (limiter == CATO_LIM_MLP5 ? 5 : 0);
}

}  // namespace cato
