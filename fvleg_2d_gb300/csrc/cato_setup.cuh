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

// reconstruction kind of a limiter id: 0 = TVD2, 3 = MLP3, 5 = MLP5
inline int recon_of_limiter(int limiter) {
  return limiter == CATO_LIM_MLP3 ? 3 : (limiter == CATO_LIM_MLP5 ? 5 : 0);
}

}  // namespace cato
