// cato_stage.cuh -- the fused RK stage kernel: ghost-cell boundary conditions, primitive
// recovery, MUSCL/MLP reconstruction, edge fluxes, flux divergence and the RK stage combine in
// one pass over HBM, with the CFL dt min-reduction and the state checks fused into the last stage.
//
// Work decomposition.  FP32: a CTA of T threads owns a strip of W = T - 2*NG output columns and
// marches over rows_per_cta rows; thread t always handles column x0 - NG + t (stage_tile_tvd for
// the TVD2 limiters, stage_tile for the others).  FP64 and double-float, whose chains are ten times
// longer: several warps per column segment, one row of edges each (edge_tile).
//
// Ghost cells are never stored: a ghost row/column index maps to its source interior cell
// (zero-gradient copy, symmetry mirror with the normal velocity negated, periodic wrap).  This
// reproduces the reference's sequential application (flux_solver.f90:138-185, zero_gradient
// full-length rows incl. corners, periodic corners only when all four sides are periodic)
// because for every valid side combination the final ghost value is that composition.
#pragma once

#include "cato_ctl.cuh"
#include "cato_physics.cuh"

namespace cato {

// How a compute type computes a stage.  Every precision keeps the same structure-of-arrays FP64
// state and FP64 stage buffers, and combines the stages (the RK accumulation) in FP64.
//   0 FP64    : reconstruction, flux and divergence in FP64 (bit-exact drop-in path)
//   1 FP32    : the stencil's conserved values rounded to FP32; reconstruction, flux and
//               divergence in FP32 (mixed)
//   2 df      : reconstruction, flux and divergence in double-float (mixed_df)
template <typename R> struct Prec;
template <> struct Prec<double> { static constexpr int kind = 0; };
template <> struct Prec<float> { static constexpr int kind = 1; };
template <> struct Prec<df> { static constexpr int kind = 2; };

struct StageArgs {
  int ni, nj, pitch;       // interior cells, row pitch (cells) of the state arrays
  int bc[4];               // by side: +x, +y, -x, -y
  int limiter;             // TVD2 limiter id (runtime)
  int rows_per_cta;
  int block;               // edge-parallel tiles: rows of a block
  int kind;                // 0: out = U_a + L*c ; 1: out = (U_a*a + U_k*b) + L*c  (each '+'
                           // flushed) ; 2: out = L (flux_solver_t%solve output, FP64 path)
  int last;                // last stage of the step: emit the CFL dt and the state checks
  double a, b, coef;       // c = coef * dt (the reference's (0.5_rk*dt), ((1/4)*dt), dt*alpha ...)
  // structure of arrays, one FP64 array per conserved variable
  const double* Uk[4];     // conserved state of this stage (stencil operand)
  const double* Ua[4];     // U_a (point-wise operand; the step's U^n)
  double* Uo[4];           // output conserved state
  const double* Pin[4];    // when non-null: primitives to use as-is for this stage (after upload)
  // device scalars
  const double* dt;
  const int* active;
  unsigned long long* dt_min;  // bits of the smallest positive dt candidate (atomicMin)
  int* status;
  // physics
  double gamma;
  double bc_p;             // outlet pressure (CATO_BC_OUTLET)
  // +x pressure input (CATO_BC_PRESSURE_INPUT): the ghost state (rho, u, p; v = 0) of rows
  // -pbc_ng .. nj+pbc_ng-1, written for this stage by pbc_edge_kernel
  const double* pbc_edge;
  int pbc_ng;
  // energy source term: q_dot_h per interior cell (pitch layout), added to the energy residual
  // (time_derivative, mod_fluid.f90:503); null without a source
  const double* src_q;
  Geom G;
};

// Source interior index of (possibly ghost) index g in [-ng, n+ng) along an axis with
// boundary types lo/hi; flip = the normal velocity component is negated (symmetry).  An
// exchange side (the rows axis of a slab only) keeps g: its ghost rows are stored below row 0
// and above row n - 1 of the slab's buffers, copied from the neighbouring slab.
__device__ __forceinline__ int map_index(int g, int n, int bc_lo, int bc_hi, bool& flip) {
  flip = false;
  if (g < 0) {
    if (bc_lo == BC_PERIODIC) return max(n + g, 0);
    if (bc_lo == BC_SYMMETRY) { flip = true; return min(-g - 1, n - 1); }
    if (bc_lo == BC_EXCHANGE) return g;
    return 0;
  }
  if (g >= n) {
    if (bc_hi == BC_PERIODIC) return min(g - n, n - 1);
    if (bc_hi == BC_SYMMETRY) { flip = true; return max(2 * n - 1 - g, 0); }
    if (bc_hi == BC_EXCHANGE) return g;
    return n - 1;
  }
  return g;
}

// Outlet ghost state on the +x side (outlet_bc.f90:101-123) from the primitives of the boundary
// cell it maps to (after the other sides' BCs, as the outlet has the lowest priority): copied
// when the boundary cell is supersonic, else the characteristic subsonic outflow state at the
// ambient pressure p_b.  The reference leaves the ghost unchanged when p_b or the boundary
// density is below tiny (p_b > 0 is enforced by the configuration check); here it keeps the copy.
template <typename R>
__device__ __forceinline__ void outlet_ghost(R gamma, R p_b, R& r, R& u, R& v, R& p) {
  const R r0 = r, p_d = p;
  if (!(p_b > Num<R>::tiny) || !(r0 > Num<R>::tiny)) return;
  const R cs = Num<R>::sqrt(gamma * rabs(Num<R>::div(p_d, r0)));
  const R vel = Num<R>::sqrt(u * u + v * v);
  const R mach = Num<R>::div(vel, cs);
  const R nx = Num<R>::div(u, vel + R(1e-30));
  const R ny = Num<R>::div(v, vel + R(1e-30));
  if (mach > R(1)) return;
  r = r0 + Num<R>::div(p_b - p_d, cs * cs);
  u = u + Num<R>::div(nx * (p_d - p_b), r0 * cs);
  v = v + Num<R>::div(ny * (p_d - p_b), r0 * cs);
  p = p_b;
}

template <int RING> __device__ __forceinline__ int slot_of(int row) {
  return (row + 4 * RING) % RING;  // rows are >= -NG
}

// Row bases of the shared-memory ring for rows center-2 .. center+3 (each row: [var][col]).
template <int RING>
__device__ __forceinline__ void ring_rows(const float* ring, int T, int center,
                                          const float* rp[6]) {
#pragma unroll
  for (int k = 0; k < 6; ++k) rp[k] = ring + slot_of<RING>(center + k - 2) * 4 * T;
}

// the flux of one edge from its left and right states; P(di, dj): the pressure of cell (i+di, j+dj)
// in reference terms, (i, j) the edge's left cell
template <typename R, int FLUX, int DIR, typename PF>
__device__ __forceinline__ void flux_of(const FluxConsts<R>& K, const Prim<R>& A, const Prim<R>& B,
                                        PF P, R F[4]) {
  if (FLUX == FLUX_AUSMPW) {
    R pc[4];
    if (DIR == 0) { pc[0] = P(0, -1); pc[1] = P(1, -1); pc[2] = P(0, 1); pc[3] = P(1, 1); }
    else { pc[0] = P(1, 0); pc[1] = P(1, 1); pc[2] = P(-1, 0); pc[3] = P(-1, 1); }
    flux_ausmpw<R, DIR>(K, A, B, pc, F);
  } else if (FLUX == FLUX_SLAU || FLUX == FLUX_SLAU2 || FLUX == FLUX_SD_SLAU ||
             FLUX == FLUX_SD_SLAU2) {
    R pa[6], pb[6];
    if (FLUX == FLUX_SD_SLAU || FLUX == FLUX_SD_SLAU2) {
      if (DIR == 0) {  // slau_solver.fypp:410-417
        pa[0] = P(0, 1);  pb[0] = P(0, 0);
        pa[1] = P(-1, 0); pb[1] = P(0, 0);
        pa[2] = P(0, -1); pb[2] = P(0, 0);
        pa[3] = P(1, -1); pb[3] = P(1, 0);
        pa[4] = P(2, 0);  pb[4] = P(1, 0);
        pa[5] = P(1, 1);  pb[5] = P(1, 0);
      } else {         // slau_solver.fypp:421-428
        pa[0] = P(-1, 0); pb[0] = P(0, 0);
        pa[1] = P(0, -1); pb[1] = P(0, 0);
        pa[2] = P(1, 0);  pb[2] = P(0, 0);
        pa[3] = P(1, 1);  pb[3] = P(0, 1);
        pa[4] = P(0, 2);  pb[4] = P(0, 1);
        pa[5] = P(-1, 1); pb[5] = P(0, 1);
      }
    }
    flux_slau<R, DIR, FLUX>(K, A, B, pa, pb, F);
  } else if (FLUX == FLUX_ROE) {
    R fa[5], fb[5];
    if (DIR == 0) {  // roe_solver.fypp:496-500
      fa[0] = P(0, 0); fb[0] = P(1, 0);
      fa[1] = P(0, 0); fb[1] = P(0, 1);
      fa[2] = P(0, 0); fb[2] = P(0, -1);
      fa[3] = P(0, 1); fb[3] = P(1, 1);
      fa[4] = P(0, -1); fb[4] = P(1, -1);
    } else {         // roe_solver.fypp:502-506
      fa[0] = P(0, 0); fb[0] = P(0, 1);
      fa[1] = P(0, 0); fb[1] = P(-1, 0);
      fa[2] = P(0, 0); fb[2] = P(1, 0);
      fa[3] = P(0, 1); fb[3] = P(-1, 1);
      fa[4] = P(0, 1); fb[4] = P(1, 1);
    }
    flux_roe<R, DIR>(K, A, B, fa, fb, F);
  } else if (FLUX == FLUX_AUSM_UP) {
    flux_ausm_up<R, DIR>(K, A, B, F);
  } else {
    flux_hllc<R, DIR>(K, A, B, F);
  }
}

// ---------------------------------------------------------------------------------------------
// one edge: reconstruct the four primitives from the ring and evaluate the flux
// ---------------------------------------------------------------------------------------------
// FP32, one copy per direction
template <int NG, int FLUX, int RECON, int DIR>
__device__ __forceinline__ void edge_flux(const float* const rp[6], int T, int lim, int col,
                                          const FluxConsts<float>& K, float F[4]) {
  // stencil sample at normal offset n and tangential offset t from the edge's left cell;
  // rp[k] is the ring row (edge row) + k - 2
  auto Q = [&](int var, int n, int t) -> float {
    return DIR == 0 ? rp[t + 2][var * T + col + n] : rp[n + 2][var * T + col + t];
  };
  float Lv[4], Rv[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (RECON == 0) {
      recon_tvd2<float>(lim, Q(k, -1, 0), Q(k, 0, 0), Q(k, 1, 0), Q(k, 2, 0), Lv[k], Rv[k]);
    } else {
      float qm2 = RECON == 5 ? Q(k, -2, 0) : 0.0f, qp3 = RECON == 5 ? Q(k, 3, 0) : 0.0f;
      recon_mlp<float, RECON>(qm2, Q(k, -1, 0), Q(k, 0, 0), Q(k, 1, 0), Q(k, 2, 0), qp3,
                              Q(k, 0, 1), Q(k, 0, -1), Q(k, 1, 1), Q(k, 1, -1), Lv[k], Rv[k]);
    }
  }
  Prim<float> A = {Lv[0], Lv[1], Lv[2], Lv[3]}, B = {Rv[0], Rv[1], Rv[2], Rv[3]};
  // cell pressures in reference (i, j) terms: P(di, dj) = p(i+di, j+dj), (i, j) = left cell
  auto P = [&](int di, int dj) -> float { return DIR == 0 ? Q(3, di, dj) : Q(3, dj, di); };
  if constexpr (FLUX == FLUX_M_AUSMPW) {
    float pc[4];
    if (DIR == 0) { pc[0] = P(0, -1); pc[1] = P(1, -1); pc[2] = P(0, 1); pc[3] = P(1, 1); }
    else { pc[0] = P(1, 0); pc[1] = P(1, 1); pc[2] = P(-1, 0); pc[3] = P(-1, 1); }
    // the superbee edge states of the second interpolator (m_ausmpw_plus_solver.fypp:163-167)
    float Ls[4], Rs[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      recon_tvd2<float>(LIM_SUPERBEE, Q(k, -1, 0), Q(k, 0, 0), Q(k, 1, 0), Q(k, 2, 0), Ls[k], Rs[k]);
    Prim<float> As = {Ls[0], Ls[1], Ls[2], Ls[3]}, Bs = {Rs[0], Rs[1], Rs[2], Rs[3]};
    flux_mausmpw<float, DIR>(K, A, B, As, Bs, pc, F);
  } else {
    flux_of<float, FLUX, DIR>(K, A, B, P, F);
  }
}

// FP64 and double-float: one copy for both directions, which halves the code (these kernels are
// sensitive to the instruction cache).  y: an edge along j; prim: shared memory, ro[k]: offset of
// this column in row (edge row) + k - 2; a variable is T apart.
template <int RECON>
__device__ __forceinline__ EdgePair recon_edge(int lim, const double q[10]) {
  if constexpr (RECON == 0) return recon_tvd2_f64(lim, q[1], q[2], q[3], q[4]);
  else
    return recon_mlp_f64<RECON>(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7], q[8], q[9]);
}
template <int RECON> __device__ __forceinline__ DfPair recon_edge(int lim, const df q[10]) {
  if constexpr (RECON == 0) return recon_tvd2_df(lim, q[1], q[2], q[3], q[4]);
  else
    return recon_mlp_df_ool<RECON>(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7], q[8], q[9]);
}
// the left and right state of variable k
template <typename R, int RECON>
__device__ __forceinline__ void edge_states(const R* prim, const int ro[6], int T, int lim, bool y,
                                            int k, R& L, R& Rr) {
  // the sample n cells along and t cells across the edge normal
  auto Q = [&](int n, int t) -> R { return prim[(y ? ro[n + 2] + t : ro[t + 2] + n) + k * T]; };
  R q[10];
  q[1] = Q(-1, 0);
  q[2] = Q(0, 0);
  q[3] = Q(1, 0);
  q[4] = Q(2, 0);
  q[0] = RECON == 5 ? Q(-2, 0) : R(0);
  q[5] = RECON == 5 ? Q(3, 0) : R(0);
  if constexpr (RECON != 0) {
    q[6] = Q(0, 1);
    q[7] = Q(0, -1);
    q[8] = Q(1, 1);
    q[9] = Q(1, -1);
  }
  const auto e = recon_edge<RECON>(lim, q);
  L = e.L;
  Rr = e.R;
}
// the flux from the states Lv, Rv in the edge's frame: u and v are exchanged before, and the
// momentum fluxes after
template <typename R, int FLUX>
__device__ __forceinline__ void edge_flux_any(const R* prim, const int ro[6], int T, bool y,
                                              const R Lv[4], const R Rv[4],
                                              const FluxConsts<R>& K, R F[4]) {
  const Prim<R> A = {Lv[0], y ? Lv[2] : Lv[1], y ? Lv[1] : Lv[2], Lv[3]};
  const Prim<R> B = {Rv[0], y ? Rv[2] : Rv[1], y ? Rv[1] : Rv[2], Rv[3]};
  // cell pressures n along and t across the normal, with t counted so that the reference's lists
  // (ausmpw_plus_solver.fypp:430-442, slau_solver.fypp:410-428) come out in their order
  [[maybe_unused]] auto P = [&](int n, int t) -> R {
    return prim[(y ? ro[n + 2] - t : ro[t + 2] + n) + 3 * T];
  };
  R G[4];
  if constexpr (FLUX == FLUX_AUSMPW) {
    const R pc[4] = {P(0, -1), P(1, -1), P(0, 1), P(1, 1)};
    flux_ausmpw<R, 0>(K, A, B, pc, G);
  } else if constexpr (FLUX == FLUX_M_AUSMPW) {
    const R pc[4] = {P(0, -1), P(1, -1), P(0, 1), P(1, 1)};
    // the superbee edge states of the second interpolator (m_ausmpw_plus_solver.fypp:163-167)
    R Ls[4], Rs[4];
#pragma unroll 1
    for (int k = 0; k < 4; ++k) edge_states<R, 0>(prim, ro, T, LIM_SUPERBEE, y, k, Ls[k], Rs[k]);
    const Prim<R> As = {Ls[0], y ? Ls[2] : Ls[1], y ? Ls[1] : Ls[2], Ls[3]};
    const Prim<R> Bs = {Rs[0], y ? Rs[2] : Rs[1], y ? Rs[1] : Rs[2], Rs[3]};
    flux_mausmpw<R, 0>(K, A, B, As, Bs, pc, G);
  } else if constexpr (FLUX == FLUX_SD_SLAU || FLUX == FLUX_SD_SLAU2) {
    const R l = P(0, 0), r = P(1, 0);
    const R pa[6] = {P(0, 1), P(-1, 0), P(0, -1), P(1, -1), P(2, 0), P(1, 1)};
    const R pb[6] = {l, l, l, r, r, r};
    flux_slau<R, 0, FLUX>(K, A, B, pa, pb, G, y);
  } else if constexpr (FLUX == FLUX_SLAU || FLUX == FLUX_SLAU2) {
    const R none[6] = {};
    flux_slau<R, 0, FLUX>(K, A, B, none, none, G, y);
  } else if constexpr (FLUX == FLUX_ROE) {
    // roe_solver.fypp:496-506; the last two pairs differ between the directions
    const R l = P(0, 0), r = P(1, 0), lp = P(0, 1), lm = P(0, -1), rp = P(1, 1), rm = P(1, -1);
    const R fa[5] = {l, l, l, y ? r : lp, y ? r : lm};
    const R fb[5] = {r, lp, lm, rp, rm};
    flux_roe<R, 0>(K, A, B, fa, fb, G, y);
  } else if constexpr (FLUX == FLUX_AUSM_UP) {
    flux_ausm_up<R, 0>(K, A, B, G);
  } else {
    flux_hllc<R, 0>(K, A, B, G);
  }
  F[0] = G[0];
  F[1] = y ? G[2] : G[1];
  F[2] = y ? G[1] : G[2];
  F[3] = G[3];
}

// ---------------------------------------------------------------------------------------------
// primitive row load
// ---------------------------------------------------------------------------------------------
template <typename R> struct RowSrc {
  double c[4];  // conserved state of the stage (or the raw primitives) as loaded
  bool flipy;
};

template <typename R>
__device__ __forceinline__ void load_src(const StageArgs& A, int sx, int row, RowSrc<R>& s) {
  bool fy;
  const int sy = map_index(row, A.nj, A.bc[SIDE_MY], A.bc[SIDE_PY], fy);
  s.flipy = fy;
  const size_t idx = (size_t)sy * A.pitch + sx;
  const double* const* src = A.Pin[0] ? A.Pin : A.Uk;
#pragma unroll
  for (int k = 0; k < 4; ++k) s.c[k] = load_global(src[k] + idx);
}

template <typename R> __device__ __forceinline__ R from_double(double x);
template <> __device__ __forceinline__ double from_double<double>(double x) { return x; }
template <> __device__ __forceinline__ float from_double<float>(double x) { return d2f_int(x); }
template <> __device__ __forceinline__ df from_double<df>(double x) { return to_df(x); }

// xmode: 0 interior / mapped ghost, 1 +x outlet ghost column, 2 +x pressure-input ghost column;
// row: the (possibly ghost) row of the sample
template <typename R>
__device__ __forceinline__ void src_to_prim(const StageArgs& A, const RowSrc<R>& s, bool flipx,
                                            int xmode, int row, R g, R g1, R out[4]) {
  if (xmode == 2) {  // lowest-priority BC: the row's edge state replaces the mapped value
    const double* e = A.pbc_edge + 3 * (size_t)(row + A.pbc_ng);
    out[0] = from_double<R>(e[0]);
    out[1] = from_double<R>(e[1]);
    out[2] = R(0);
    out[3] = from_double<R>(e[2]);
    return;
  }
  R r, u, v, p;
  if constexpr (Prec<R>::kind == 0) {
    if (A.Pin[0]) {
      r = s.c[0]; u = s.c[1]; v = s.c[2]; p = s.c[3];
    } else {
      R cs;
      r = s.c[0];
      prim_from_cons(g, g1, r, s.c[1], s.c[2], s.c[3], u, v, p, cs);
    }
  } else if constexpr (Prec<R>::kind == 2) {
    if (A.Pin[0]) {
      r = to_df(s.c[0]); u = to_df(s.c[1]); v = to_df(s.c[2]); p = to_df(s.c[3]);
    } else {
      R cs;
      r = to_df(s.c[0]);
      const df rE = to_df(s.c[3]);
      prim_from_cons(g, g1, r, to_df(s.c[1]), to_df(s.c[2]), rE, u, v, p, cs, false);
      if (near_vacuum(p.hi, rE.hi, 1e-4f)) {
        double u64, v64, p64;
        prim_from_cons_f64(A.gamma, s.c[0], s.c[1], s.c[2], s.c[3], u64, v64, p64);
        u = to_df(u64); v = to_df(v64); p = to_df(p64);
      }
    }
  } else {
    r = d2f_fast(s.c[0]);
    if (A.Pin[0]) {
      u = d2f_fast(s.c[1]); v = d2f_fast(s.c[2]); p = d2f_fast(s.c[3]);
    } else {
      R cs;
      prim_from_cons(g, g1, r, d2f_fast(s.c[1]), d2f_fast(s.c[2]), d2f_fast(s.c[3]), u, v, p,
                     cs);
    }
  }
  u = flipx ? rneg(u) : u;
  v = s.flipy ? rneg(v) : v;
  if (xmode == 1) outlet_ghost<R>(g, R(A.bc_p), r, u, v, p);
  out[0] = r;
  out[1] = u;
  out[2] = v;
  out[3] = p;
}

// ---------------------------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------------------------
// What a thread keeps for its column during a tile.
template <typename R> struct ColumnConsts {
  double cc;  // coef * dt
  float ccf, cfl_f;        // mixed: the stage increment c L in FP32
  float idx_col, idy_uni;  // FP32 reciprocal cell width of the column / row height (uniform grid)
  df dx_inv, dy_inv, cfl_df, cc_df;  // mixed_df constants of the update
  double dt_loc;           // smallest CFL dt and status bits of the column's new states
  int st_loc;

  // (the constants come converted with the scheme's: their FP64 divisions and conversions, per
  // thread, were a quarter of the double-float kernel's FP64-pipe work)
  template <bool EXT>
  __device__ __forceinline__ void init(const StageArgs& A, const FluxConsts<R>& K, int gx) {
    cc = A.coef * *A.dt;
    if constexpr (Prec<R>::kind == 2) {
      dx_inv = A.G.rdxc ? to_df(A.G.rdxc[min(max(gx, 0), A.ni - 1)]) : K.rdx;
      dy_inv = K.rdy;
      cfl_df = K.cfl;
      cc_df = to_df(cc);
    }
    if constexpr (Prec<R>::kind == 1) {
      ccf = (float)cc;
      cfl_f = K.cfl;
      idx_col = (EXT && A.G.rdxf) ? A.G.rdxf[min(max(gx, 0), A.ni - 1)] : K.rdx;
      idy_uni = K.rdy;
    }
    dt_loc = INFINITY;
    st_loc = 0;
  }
  // mixed_df on a rectilinear grid: the reciprocal height of row j
  __device__ __forceinline__ void set_row(const StageArgs& A, int j) {
    if (A.G.rdyc) dy_inv = to_df(A.G.rdyc[j]);
  }
};

// The operands of a cell's stage combine.
__device__ __forceinline__ void load_operands(const StageArgs& A, size_t cidx, double ua[4],
                                              double uk[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    ua[k] = A.Ua[k] ? A.Ua[k][cidx] : 0.0;  // may alias Uo: plain load, read before write
    uk[k] = (A.kind == 1) ? load_global(A.Uk[k] + cidx) : 0.0;
  }
}

// (out of line, so that the compiler branches to it instead of adding under a predicate)
static __device__ __noinline__ double add_source(double L, double q) { return L + q; }
static __device__ __noinline__ double scaled_source(df L, double q, double c) {
  return __dmul_rn(from_df(L) + q, c);
}

// FP64 and double-float: the divergence of variable k of a cell and its stage combine, from the
// fluxes of the cell's right, left, upper and lower edge.
template <typename R>
__device__ __forceinline__ double combine_var(const StageArgs& A, const ColumnConsts<R>& C,
                                              [[maybe_unused]] const Geom& cg,
                                              [[maybe_unused]] const Rcp<double>& vol, int k,
                                              size_t cidx, double ua, double uk, R Fi, R Fim, R Fj,
                                              R Fjm) {
  double r;
  if constexpr (Prec<R>::kind == 0) {
    double L = divergence_fp64(Fi, Fim, Fj, Fjm, cg, vol);
    if (k == 3 && A.src_q) L = add_source(L, A.src_q[cidx]);
    if (A.kind == 2) {
      r = L;
    } else if (A.kind == 0) {
      r = ua + __dmul_rn(L, C.cc);
      if (abs_lt(r, Num<double>::eps)) r = 0.0;
    } else {
      double s = __dmul_rn(ua, A.a) + __dmul_rn(uk, A.b);
      if (abs_lt(s, Num<double>::eps)) s = 0.0;
      r = s + __dmul_rn(L, C.cc);
      if (abs_lt(r, Num<double>::eps)) r = 0.0;
    }
  } else {
    // double-float divergence (pairs on the FP32 pipe) carried to FP64 once; the RK
    // accumulation in FP64: U^n + c L, or a U^n + b U^k + c L as two FP64 FMAs with the
    // increment c L formed in double-float: three FP64 operations per variable instead
    // of six (stages 2 and 3 of SSP-RK3 on the 4096^2 quadrant: 6 % faster)
    const df Ld = -((Fi - Fim) * C.dx_inv + (Fj - Fjm) * C.dy_inv);
    const bool src = k == 3 && A.src_q;
    if (A.kind == 2) {
      r = from_df(Ld);
      if (src) r = add_source(r, A.src_q[cidx]);
    } else if (A.kind == 0) {
      double L = from_df(Ld);
      if (src) L = add_source(L, A.src_q[cidx]);
      r = ua + __dmul_rn(L, C.cc);
      if (abs_lt(r, Num<double>::eps)) r = 0.0;
    } else {
      double d;
      if (src) d = scaled_source(Ld, A.src_q[cidx], C.cc);
      else d = from_df(Ld * C.cc_df);
      r = fma(uk, A.b, fma(ua, A.a, d));
      if (abs_lt(r, Num<double>::eps)) r = 0.0;
    }
  }
  return r;
}

// The CFL dt and the checks of a cell's new state (the last stage).
template <typename R, bool EXT>
__device__ __forceinline__ void check_state(const StageArgs& A, const FluxConsts<R>& K,
                                            ColumnConsts<R>& C,
                                            [[maybe_unused]] const Geom& cg,
                                            [[maybe_unused]] int j, const double un[4]) {
  [[maybe_unused]] const R g = K.gamma, g1 = K.gm1;
  // CFL dt of the new state (get_timestep, mod_fluid.f90:554-558) and the sanity checks
  if constexpr (Prec<R>::kind == 0) {
    double u, v, p, cs;
    prim_from_cons(g, g1, un[0], un[1], un[2], un[3], u, v, p, cs);
    double d = div_rn(K.cfl, quot_rn(rabs(u) + cs, cg.dx, cg.dx_y62) +
                                  quot_rn(rabs(v) + cs, cg.dy, cg.dy_y62));
    if (d_less(d, C.dt_loc)) C.dt_loc = d;
    if (d_isnan(un[0]) || d_isnan(u) || d_isnan(v) || d_isnan(p)) C.st_loc |= ST_NAN;
    if (lt0(un[0])) C.st_loc |= ST_NEG_DENSITY;
    if (lt0(p)) C.st_loc |= ST_NEG_PRESSURE;
  } else if constexpr (Prec<R>::kind == 2) {
    df u, v, p, cs;
    const df rE = to_df(un[3]);
    prim_from_cons(g, g1, to_df(un[0]), to_df(un[1]), to_df(un[2]), rE, u, v, p, cs, true);
    if (near_vacuum(p.hi, rE.hi, 1e-4f)) {  // the FP64 recovery decides p and its sign
      double u64, v64, p64;
      prim_from_cons_f64(A.gamma, un[0], un[1], un[2], un[3], u64, v64, p64);
      u = to_df(u64); v = to_df(v64); p = to_df(p64);
      cs = df_sqrt(g * df_div(p, to_df(un[0])));
    }
    const df d = df_div(C.cfl_df, (df_abs(u) + cs) * C.dx_inv + (df_abs(v) + cs) * C.dy_inv);
    const double dd = from_df(d);
    if (dd > 0.0 && dd < C.dt_loc) C.dt_loc = dd;
    if (isnan(un[0]) || isnan(u.hi) || isnan(v.hi) || isnan(p.hi)) C.st_loc |= ST_NAN;
    if (un[0] < 0.0) C.st_loc |= ST_NEG_DENSITY;
    if (p.hi < 0.0f) C.st_loc |= ST_NEG_PRESSURE;
  } else {
    const float4 uf = make_float4(d2f_fast(un[0]), d2f_fast(un[1]), d2f_fast(un[2]),
                                  d2f_fast(un[3]));
    float u, v, p, cs;
    prim_from_cons(g, g1, uf.x, uf.y, uf.z, uf.w, u, v, p, cs);
    float d = C.cfl_f / ((fabsf(u) + cs) * C.idx_col +
                       (fabsf(v) + cs) * ((EXT && A.G.rdyf) ? A.G.rdyf[j] : C.idy_uni));
    double dd = f2d_int(d);
    if (__double_as_longlong(dd) < __double_as_longlong(C.dt_loc) && d > 0.0f) C.dt_loc = dd;
    // NaN and sign tests on the FP64 state itself (the fast conversion keeps neither)
    if (d_isnan(un[0]) || d_isnan(un[1]) || d_isnan(un[2]) || d_isnan(un[3]) ||
        isnan(u) || isnan(v) || isnan(p))
      C.st_loc |= ST_NAN;
    if (lt0(un[0])) C.st_loc |= ST_NEG_DENSITY;
    if (p < 0.0f) C.st_loc |= ST_NEG_PRESSURE;
  }
}

// FP32: one cell's divergence, stage combine and (in the last stage) CFL dt and state checks.
template <bool EXT>
__device__ __forceinline__ void update_cell(const StageArgs& A, const FluxConsts<float>& K,
                                            ColumnConsts<float>& C, int gx, int j,
                                            size_t cidx, const double ua[4], const double uk[4],
                                            const float Fi_[4], const float Fim_[4], const float Fj_[4],
                                            const float Fjm_[4]) {
  double un[4];
  // the cell's metrics (constants on a uniform grid)
  const Geom cg = cell_geom(A.G, gx, j);
  // FP32 divergence and stage increment c L; the stage combine (the RK accumulation)
  // in FP64
  const float idx_f = C.idx_col;
  const float idy_f = (EXT && A.G.rdyf) ? A.G.rdyf[j] : C.idy_uni;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float Fi = Fi_[k], Fim = Fim_[k], Fj = Fj_[k], Fjm = Fjm_[k];
    float Lf = -((Fi - Fim) * idx_f + (Fj - Fjm) * idy_f);
    if (EXT && k == 3 && A.src_q) Lf = Lf + d2f_int(A.src_q[cidx]);
    double r;
    if (A.kind == 2) r = f2d_int(Lf);
    else if (A.kind == 0) r = ua[k] + f2d_int(Lf * C.ccf);
    else r = fma(uk[k], A.b, fma(ua[k], A.a, f2d_int(Lf * C.ccf)));
    un[k] = r;
    A.Uo[k][cidx] = r;
  }
  if (A.last) check_state<float, EXT>(A, K, C, cg, j, un);
}

// The column's CFL dt and status into the step control.
template <typename R>
__device__ __forceinline__ void reduce_column(const StageArgs& A, const ColumnConsts<R>& C) {
  double dt_loc = C.dt_loc;
  int st_loc = C.st_loc;
  const int t = threadIdx.x;
  if (!A.last) return;
  // block min of dt (bits of positive doubles order as unsigned integers) and status OR
  unsigned long long bits =
      (dt_loc > 0.0) ? (unsigned long long)__double_as_longlong(dt_loc) : ~0ULL;
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long ob = __shfl_xor_sync(0xffffffffu, bits, o);
    bits = ob < bits ? ob : bits;
    st_loc |= __shfl_xor_sync(0xffffffffu, st_loc, o);
  }
  if ((t & 31) == 0) {
    if (bits != ~0ULL) atomicMin(A.dt_min, bits);
    if (st_loc) atomicOr(A.status, st_loc);
  }
}

// How a column's samples are made: 0 interior / mapped ghost, 1 +x outlet ghost column, 2 +x
// pressure-input ghost column (the lowest-priority BCs).
template <bool EXT> __device__ __forceinline__ int column_mode(const StageArgs& A, int gx) {
  return gx < A.ni ? 0
         : A.bc[SIDE_PX] == BC_OUTLET
             ? 1
             : (EXT && A.bc[SIDE_PX] == BC_PRESSURE_INPUT ? 2 : 0);
}

// FP32: one tile: columns [bx*W, bx*W + W) x rows [by*rows_per_cta, ...) of one instance.
// EXT = false compiles out the rectilinear metrics, the energy source and the pressure-input
// ghost columns (a uniform grid without them); the issue-bound FP32 path uses it whenever it can.
template <int NG, int FLUX, int RECON, bool EXT>
__device__ __forceinline__ void stage_tile(const StageArgs& A, const FluxConsts<float>& K, int bx,
                                           int by, unsigned char* smem_raw) {
  using R = float;
  constexpr int RING = 2 * NG;
  const int T = blockDim.x, W = T - 2 * NG, t = threadIdx.x;
  const int x0 = bx * W;
  const int gx = x0 - NG + t;
  const int y0 = by * A.rows_per_cta;
  const int y1 = min(y0 + A.rows_per_cta, A.nj);
  R* ring = reinterpret_cast<R*>(smem_raw);  // [RING][4][T]
  R* sfi = ring + RING * 4 * T;              // [4][T]   i-edge between cols t and t+1
  R* sfj = sfi + 4 * T;                      // [2][4][T] j-edge between rows j and j+1 at slot j&1

  const R g = K.gamma, g1 = K.gm1;
  bool flipx;
  const int sx = map_index(min(gx, A.ni + NG - 1), A.ni, A.bc[SIDE_MX], A.bc[SIDE_PX], flipx);
  const int xmode = column_mode<EXT>(A, gx);
  const bool in_i_edge = (t >= NG - 1) && (t <= NG + W - 1) && (gx <= A.ni - 1);
  const bool in_cell = (t >= NG) && (t <= NG + W - 1) && (gx < A.ni);
  ColumnConsts<R> C;
  C.template init<EXT>(A, K, gx);
  const R* rp[6];

  // prologue: rows y0-NG .. y0+NG-1
  for (int r = y0 - NG; r < y0 + NG; ++r) {
    RowSrc<R> s;
    load_src<R>(A, sx, r, s);
    R q[4];
    src_to_prim<R>(A, s, flipx, xmode, r, g, g1, q);
    R* row = ring + slot_of<RING>(r) * 4 * T;
#pragma unroll
    for (int k = 0; k < 4; ++k) row[k * T + t] = q[k];
  }
  __syncthreads();
  if (in_cell && y0 < y1) {
    R F[4];
    ring_rows<RING>(ring, T, y0 - 1, rp);
    edge_flux<NG, FLUX, RECON, 1>(rp, T, A.limiter, t, K, F);
#pragma unroll
    for (int k = 0; k < 4; ++k) sfj[(((y0 - 1) & 1) * 4 + k) * T + t] = F[k];
  }
  __syncthreads();

  RowSrc<R> pre;
  if (y0 < y1) load_src<R>(A, sx, y0 + NG, pre);

  for (int j = y0; j < y1; ++j) {
    // operands of this row's cell update, issued early
    const size_t cidx = (size_t)j * A.pitch + (size_t)min(max(gx, 0), A.ni - 1);
    double ua[4], uk[4];
    if (in_cell) load_operands(A, cidx, ua, uk);
    RowSrc<R> nxt;
    if (j + 1 < y1) load_src<R>(A, sx, j + 1 + NG, nxt);
    {
      R q[4];
      src_to_prim<R>(A, pre, flipx, xmode, j + NG, g, g1, q);
      R* row = ring + slot_of<RING>(j + NG) * 4 * T;
#pragma unroll
      for (int k = 0; k < 4; ++k) row[k * T + t] = q[k];
    }
    pre = nxt;
    __syncthreads();
    ring_rows<RING>(ring, T, j, rp);
    if (in_i_edge) {
      R F[4];
      edge_flux<NG, FLUX, RECON, 0>(rp, T, A.limiter, t, K, F);
#pragma unroll
      for (int k = 0; k < 4; ++k) sfi[k * T + t] = F[k];
    }
    if (in_cell) {
      R F[4];
      edge_flux<NG, FLUX, RECON, 1>(rp, T, A.limiter, t, K, F);
#pragma unroll
      for (int k = 0; k < 4; ++k) sfj[((j & 1) * 4 + k) * T + t] = F[k];
    }
    __syncthreads();
    if (in_cell) {
      R Fi[4], Fim[4], Fj[4], Fjm[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        Fi[k] = sfi[k * T + t];
        Fim[k] = sfi[k * T + t - 1];
        Fj[k] = sfj[((j & 1) * 4 + k) * T + t];
        Fjm[k] = sfj[(((j - 1) & 1) * 4 + k) * T + t];
      }
      update_cell<EXT>(A, K, C, gx, j, cidx, ua, uk, Fi, Fim, Fj, Fjm);
    }
  }
  reduce_column(A, C);
}

// ---------------------------------------------------------------------------------------------
// the TVD2 tile
// ---------------------------------------------------------------------------------------------
// Whether a flux reads cell pressures around the edge (shock sensors).
constexpr bool flux_reads_pressure(int flux) {
  return flux == FLUX_AUSMPW || flux == FLUX_SD_SLAU || flux == FLUX_SD_SLAU2 || flux == FLUX_ROE;
}
// M-AUSMPW+ reconstructs twice per edge (its second interpolator) and keeps the general tile.
constexpr bool tvd_tile_of(int flux, int recon) { return recon == 0 && flux != FLUX_M_AUSMPW; }
// rows of primitives it keeps
constexpr int tvd_ring_rows(int flux) { return flux_reads_pressure(flux) ? 4 : 2; }

// Edge values of N cells from their lower and upper differences: L the left state of the edge
// above, Rr the right state of the edge below.  phi(b / a) a is symmetric in a and b for every
// TVD2 limiter, so one limited slope serves both.  One limiter choice for all N cells, so that
// their slopes stand in one block.
template <int N>
__device__ __forceinline__ void tvd_cells(int lim, const float q[N], const float a[N],
                                          const float b[N], float L[N], float Rr[N]) {
  auto all = [&](auto lc) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const float s = tvd_slope_f32(decltype(lc)::value, b[k], a[k]);
      L[k] = q[k] + 0.5f * s;
      Rr[k] = q[k] - 0.5f * s;
    }
  };
  if (lim == LIM_MINMOD) all(std::integral_constant<int, LIM_MINMOD>{});
  else if (lim == LIM_SUPERBEE) all(std::integral_constant<int, LIM_SUPERBEE>{});
  else all(std::integral_constant<int, LIM_VANLEER>{});
}

// One tile of a TVD2 scheme (FP32).  A cell's two edge values along a direction come from the same
// two differences and one limited slope, so they are made once per cell (the edge-wise form makes
// every difference three times and every slope twice), and the march keeps what the next row needs
// in registers: the lower difference and the upper left state of the column, the right-hand left
// state of the row, the fluxes of the edge below.  Shared memory only carries what the
// neighbouring columns read: the row of primitives (a ring of 4 rows where the flux reads
// pressures around the edge, else 2), the right states and the x fluxes, each double-buffered by
// row, so that one __syncthreads per row orders them all.
//
// Row j of the march: row j + 2 enters; the y values of cell j + 1 complete edge j + 1/2; the x
// fluxes of row j use the values of the row before; the x values of row j + 1; barrier; update.
template <int FLUX, bool EXT>
__device__ __forceinline__ void stage_tile_tvd(const StageArgs& A, const FluxConsts<float>& K,
                                               int bx, int by, unsigned char* smem_raw) {
  constexpr int NG = 2, RR = tvd_ring_rows(FLUX);
  const int T = blockDim.x, W = T - 2 * NG, t = threadIdx.x;
  const int gx = bx * W - NG + t;
  const int y0 = by * A.rows_per_cta;
  const int y1 = min(y0 + A.rows_per_cta, A.nj);
  float* const ring = reinterpret_cast<float*>(smem_raw);  // [RR][4][T] row r at slot r % RR
  float* const srm = ring + RR * 4 * T;  // [2][4][T] right state of the cell's left edge
  float* const sfi = srm + 8 * T;        // [2][4][T] flux of the edge right of the cell
  auto row_at = [&](int r) { return ring + ((r + RR) & (RR - 1)) * 4 * T; };

  const float g = K.gamma, g1 = K.gm1;
  bool flipx;
  const int sx = map_index(min(gx, A.ni + NG - 1), A.ni, A.bc[SIDE_MX], A.bc[SIDE_PX], flipx);
  const int xmode = column_mode<EXT>(A, gx);
  const bool in_x = t >= 1 && t <= T - 2 && gx <= A.ni;  // columns whose x values are read
  const bool in_cell = t >= NG && t <= NG + W - 1 && gx < A.ni;
  ColumnConsts<float> C;
  C.template init<EXT>(A, K, gx);

  auto prims_of = [&](const RowSrc<float>& src, int row, float q[4]) {
    src_to_prim<float>(A, src, flipx, xmode, row, g, g1, q);
  };
  auto store_row = [&](int r, const float q[4]) {
    float* row = row_at(r);
#pragma unroll
    for (int k = 0; k < 4; ++k) row[k * T + t] = q[k];
  };
  auto flux_y = [&](int j, const float L[4], const float Rr[4], float F[4]) {
    auto P = [&](int di, int dj) -> float { return row_at(j + dj)[3 * T + t + di]; };
    flux_of<float, FLUX, 1>(K, {L[0], L[1], L[2], L[3]}, {Rr[0], Rr[1], Rr[2], Rr[3]}, P, F);
  };
  auto flux_x = [&](int j, const float L[4], float F[4]) {
    auto P = [&](int di, int dj) -> float { return row_at(j + dj)[3 * T + t + di]; };
    const float* rm = srm + (j & 1) * 4 * T + t + 1;
    flux_of<float, FLUX, 0>(K, {L[0], L[1], L[2], L[3]}, {rm[0], rm[T], rm[2 * T], rm[3 * T]}, P, F);
  };

  float q1[4], a[4], Lt[4], Lx[4], Fb[4];  // row j + 1, its lower difference; carried values
  RowSrc<float> pre;
  // rows y0-2 .. y0+1, the y values of cells y0-1 and y0, the flux of edge y0-1/2, the x values
  // of row y0
  {
    float q[4][4], d[3][4], Rt[4], Rb[4], L1[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      load_src<float>(A, sx, y0 - 2 + r, pre);
      prims_of(pre, y0 - 2 + r, q[r]);
      if (r >= 4 - RR) store_row(y0 - 2 + r, q[r]);
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int k = 0; k < 4; ++k) d[r][k] = q[r + 1][k] - q[r][k];
    if (in_cell) {
      tvd_cells<4>(A.limiter, q[1], d[0], d[1], Lt, Rt);
      tvd_cells<4>(A.limiter, q[2], d[1], d[2], L1, Rb);
    }
    __syncthreads();
    if (in_cell) {
      flux_y(y0 - 1, Lt, Rb, Fb);
#pragma unroll
      for (int k = 0; k < 4; ++k) Lt[k] = L1[k];
    }
    if (in_x) {
      const float* row = row_at(y0);
      float lo[4], up[4], Rm[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        lo[k] = q[2][k] - row[k * T + t - 1];
        up[k] = row[k * T + t + 1] - q[2][k];
      }
      tvd_cells<4>(A.limiter, q[2], lo, up, Lx, Rm);
#pragma unroll
      for (int k = 0; k < 4; ++k) srm[((y0 & 1) * 4 + k) * T + t] = Rm[k];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      q1[k] = q[3][k];
      a[k] = d[2][k];
    }
  }
  if (y0 < y1) load_src<float>(A, sx, y0 + 2, pre);
  __syncthreads();

  for (int j = y0; j < y1; ++j) {
    const size_t cidx = (size_t)j * A.pitch + (size_t)min(max(gx, 0), A.ni - 1);
    double ua[4], uk[4];
    if (in_cell) load_operands(A, cidx, ua, uk);
    float q2[4], Ft[4];
    prims_of(pre, j + 2, q2);
    if (j + 1 < y1) load_src<float>(A, sx, j + 3, pre);
    store_row(j + 2, q2);
    // one block for both directions (columns without a cell compute values nobody reads), so that
    // the two chains overlap
    if (in_x) {
      const float* row = row_at(j + 1);
      float q[8], lo[8], up[8], Lv[8], Rv[8], F[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        q[k] = q[4 + k] = q1[k];
        lo[k] = a[k];
        up[k] = q2[k] - q1[k];
        lo[4 + k] = q1[k] - row[k * T + t - 1];
        up[4 + k] = row[k * T + t + 1] - q1[k];
      }
      tvd_cells<8>(A.limiter, q, lo, up, Lv, Rv);
      flux_y(j, Lt, Rv, Ft);
      flux_x(j, Lx, F);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        sfi[((j & 1) * 4 + k) * T + t] = F[k];
        srm[(((j + 1) & 1) * 4 + k) * T + t] = Rv[4 + k];
        a[k] = up[k];
        Lt[k] = Lv[k];
        Lx[k] = Lv[4 + k];
        q1[k] = q2[k];
      }
    }
    __syncthreads();
    if (in_cell) {
      float Fi[4], Fim[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        Fi[k] = sfi[((j & 1) * 4 + k) * T + t];
        Fim[k] = sfi[((j & 1) * 4 + k) * T + t - 1];
      }
      update_cell<EXT>(A, K, C, gx, j, cidx, ua, uk, Fi, Fim, Ft, Fb);
#pragma unroll
      for (int k = 0; k < 4; ++k) Fb[k] = Ft[k];
    }
  }
  reduce_column(A, C);
}

// ---------------------------------------------------------------------------------------------
// the edge-parallel tile
// ---------------------------------------------------------------------------------------------
// Several warps (warp pairs with T = 64) on a segment of T columns incl. the x-halo: blockDim =
// (T, nw), nw >= 2 RW + 1.  The tile marches in blocks of RW rows.  Per block RW new rows of
// primitives enter a ring of RW + 2 NG rows; then every warp makes one row of edges, RW + 1 rows
// of y edges (RW after the first block, whose lower row is carried) and RW rows of x edges side by
// side; then all warps share the (cell, variable) updates, with a barrier after each phase.  The
// serial chain of a block is one edge, against a row's two edges and update in the marching strip,
// and a CTA has 2 RW + 1 times the warps for the same columns, so that the latency of the long
// FP64 chains is covered with few registers per thread.
//
// SPLIT, for grids that leave SMs idle: the states of an edge row are made by one warp per
// variable and handed over in shared memory, and nw may be larger, so that the chain is one
// variable's states, one flux and one update (FP64 64 x 48: 75 -> 55 us a step; where the GPU is
// full the hand-over costs 3 % in FP64 and 7 % in double-float).
struct EdgeShape {
  int columns;  // T
  int block;    // RW
  int warps;    // nw: 2 RW + 1, or more for the split form
  constexpr bool split() const { return warps > 2 * block + 1; }
};
template <typename R, int NG, int FLUX, int RECON, bool SPLIT>
__device__ __forceinline__ void edge_tile(const StageArgs& A, const FluxConsts<R>& K, int bx,
                                          int by, unsigned char* smem_raw) {
  const int T = blockDim.x, nw = blockDim.y, RW = A.block, NR = RW + 2 * NG, NE = 2 * RW + 1;
  const int t = threadIdx.x, w = threadIdx.y;
  const int gx = bx * (T - 2 * NG) - NG + t;
  const int y0 = by * A.rows_per_cta, y1 = min(y0 + A.rows_per_cta, A.nj);
  double* const un = reinterpret_cast<double*>(smem_raw);  // [RW][4][T] new states
  R* const prim = reinterpret_cast<R*>(un + RW * 4 * T);   // [NR][4][T] row r at slot (r - y0 + NG) % NR
  R* const sfx = prim + NR * 4 * T;                        // [RW][4][T] edge right of the cell
  R* const sfy = sfx + RW * 4 * T;                         // [RW + 1][4][T] edge above row e at
                                                           // slot (e - y0 + 1) % (RW + 1)
  R* const st = sfy + (RW + 1) * 4 * T;                    // SPLIT: [NE][4][2][T] left and right states
  const R g = K.gamma, g1 = K.gm1;
  bool flipx;
  const int sx = map_index(min(gx, A.ni + NG - 1), A.ni, A.bc[SIDE_MX], A.bc[SIDE_PX], flipx);
  const int xmode = column_mode<true>(A, gx);
  const bool in_i_edge = t >= NG - 1 && t < T - NG && gx <= A.ni - 1;
  const bool in_cell = t >= NG && t < T - NG && gx < A.ni;
  ColumnConsts<R> C;
  C.template init<true>(A, K, gx);

  int next = -NG;  // first row (relative to y0) not yet in the ring
  for (int yb = y0; yb < y1; yb += RW) {
    const int rows = min(RW, y1 - yb);
    const int upto = yb - y0 + rows + NG;  // rows below this one are needed
    for (int r = next + w; r < upto; r += nw) {
      RowSrc<R> s;
      load_src<R>(A, sx, y0 + r, s);
      R q[4];
      src_to_prim<R>(A, s, flipx, xmode, y0 + r, g, g1, q);
      R* row = prim + (r + NG) % NR * 4 * T;
#pragma unroll
      for (int k = 0; k < 4; ++k) row[k * T + t] = q[k];
    }
    next = upto;
    __syncthreads();
    // edge row m: the y edges above row yb - 1 + m for m <= RW, else the x edges of row
    // yb + m - RW - 1; none beyond the tile, and m = 0 only in the first block
    auto edge_row = [&](int m) { return m <= RW ? yb - 1 + m : yb + m - RW - 1; };
    auto edge_on = [&](int m) { return edge_row(m) < y1 && (m > 0 || yb == y0); };
    // this column in rows e - 2 .. e + 3 (NG = 2 reads e - 1 .. e + 2)
    auto rows_of = [&](int e, int ro[6]) {
      int slot = (e - y0 + NG - 2 + NR) % NR;
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        ro[k] = slot * 4 * T + t;
        slot = slot + 1 == NR ? 0 : slot + 1;
      }
    };
    if constexpr (SPLIT) {
      for (int n = w; n < NE * 4; n += nw) {
        const int m = n >> 2, k = n & 3;
        const bool along_y = m <= RW;
        if (!edge_on(m) || !(along_y ? in_cell : in_i_edge)) continue;
        int ro[6];
        rows_of(edge_row(m), ro);
        R L, Rr;
        edge_states<R, RECON>(prim, ro, T, A.limiter, along_y, k, L, Rr);
        st[(2 * n) * T + t] = L;
        st[(2 * n + 1) * T + t] = Rr;
      }
      __syncthreads();
    }
    if (w < NE && edge_on(w)) {
      const bool along_y = w <= RW;
      if (along_y ? in_cell : in_i_edge) {
        const int e = edge_row(w);
        int ro[6];
        rows_of(e, ro);
        R L[4], Rr[4], F[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if constexpr (SPLIT) {
            L[k] = st[(8 * w + 2 * k) * T + t];
            Rr[k] = st[(8 * w + 2 * k + 1) * T + t];
          } else {
            edge_states<R, RECON>(prim, ro, T, A.limiter, along_y, k, L[k], Rr[k]);
          }
        }
        edge_flux_any<R, FLUX>(prim, ro, T, along_y, L, Rr, K, F);
        R* out = along_y ? sfy + (e - y0 + 1) % (RW + 1) * 4 * T : sfx + (e - yb) * 4 * T;
#pragma unroll
        for (int k = 0; k < 4; ++k) out[k * T + t] = F[k];
      }
    }
    __syncthreads();
    for (int n = w; n < rows * 4; n += nw) {
      if (!in_cell) continue;
      const int r = n >> 2, k = n & 3, j = yb + r;
      const size_t cidx = (size_t)j * A.pitch + gx;
      const Geom cg = cell_geom(A.G, gx, j);
      if constexpr (Prec<R>::kind == 2) C.set_row(A, j);
      const double ua = A.Ua[k] ? A.Ua[k][cidx] : 0.0;
      const double uk = A.kind == 1 ? load_global(A.Uk[k] + cidx) : 0.0;
      const R* fj = sfy + ((j - y0 + 1) % (RW + 1) * 4 + k) * T + t;
      const R* fjm = sfy + ((j - y0) % (RW + 1) * 4 + k) * T + t;
      const double u = combine_var<R>(A, C, cg, Rcp<double>(cg.vol, cg.vol_y62), k, cidx, ua, uk,
                                      sfx[n * T + t], sfx[n * T + t - 1], *fj, *fjm);
      A.Uo[k][cidx] = u;
      if (A.last) un[n * T + t] = u;
    }
    if (!A.last) continue;
    __syncthreads();
    if (w < rows && in_cell) {
      const int j = yb + w;
      const double* v = un + w * 4 * T + t;
      const double u4[4] = {v[0], v[T], v[2 * T], v[3 * T]};
      if constexpr (Prec<R>::kind == 2) C.set_row(A, j);
      check_state<R, true>(A, K, C, cell_geom(A.G, gx, j), j, u4);
    }
  }
  if (w < RW) reduce_column(A, C);
}
template <typename R> constexpr size_t edge_smem_bytes(EdgeShape s, int ng) {
  const size_t rows = 3 * s.block + 2 * ng + 1 + (s.split() ? 2 * (2 * s.block + 1) : 0);
  return (size_t)s.columns * 4 * (sizeof(double) * s.block + sizeof(R) * rows);
}
constexpr int kEdgeThreads = 1024;  // most threads of a CTA

// ---------------------------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------------------------
// FP32: the marching strips.  The tile of a scheme, and its dynamic shared memory.
template <int NG, int FLUX, int RECON, bool EXT, bool TVD = tvd_tile_of(FLUX, RECON)>
__device__ __forceinline__ void tile_of(const StageArgs& A, const FluxConsts<float>& K, int bx,
                                        int by, unsigned char* smem_raw) {
  if constexpr (TVD) stage_tile_tvd<FLUX, EXT>(A, K, bx, by, smem_raw);
  else stage_tile<NG, FLUX, RECON, EXT>(A, K, bx, by, smem_raw);
}
constexpr size_t tile_smem_bytes(int T, int ng, int flux, bool tvd) {
  const int per_column = tvd ? tvd_ring_rows(flux) * 4 + 16 : 2 * ng * 4 + 4 + 8;
  return sizeof(float) * (size_t)T * per_column;
}
// In the persistent batch kernels AUSMPW+ keeps the general tile: there the contraction the
// assembler picks for its TVD2 tile rounds the products the other way (5e-10 of the density in 6
// steps), and a request's result would change.
constexpr bool batch_tvd_tile_of(int flux, int recon) {
  return tvd_tile_of(flux, recon) && flux != FLUX_AUSMPW;
}

// Registers per thread of the FP32 kernels.
// Single grids: HLLC, Roe and AUSM+-up with the TVD2 tile at 104 (the compiler's 113 to 135 leave
// four 128-thread CTAs on an SM; 4096^2 HLLC 1469 -> 1307 us a step), the others the compiler's
// choice, where a cap changes which products the assembler fuses and with it the rounding.  Roe
// with the rectilinear, source and pressure-input code spills at 104 and takes 128 (layered
// 1500 x 1040: 261 us a step, 287 at 104, 255 uncapped; 3000 x 2010: 765, 862 and 922).
// Batches: the general tile at 64 (+4.5 % on the batched workload), the TVD2 tile at 128.
constexpr int f32_regs(int flux, int recon, bool ext) {
  const bool capped = flux == FLUX_HLLC || flux == FLUX_ROE || flux == FLUX_AUSM_UP;
  return recon != 0 || !capped ? 255 : (ext && flux == FLUX_ROE ? 128 : 104);
}
constexpr int f32_batch_regs(int flux, int recon) {
  return batch_tvd_tile_of(flux, recon) ? 128 : 64;
}

template <int NG, int FLUX, int RECON, bool EXT>
__global__ void __maxnreg__(f32_regs(FLUX, RECON, EXT))
    stage_kernel(const StageArgs A, const FluxConsts<float> K) {
  wait_previous();
  if (A.active && *A.active == 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  tile_of<NG, FLUX, RECON, EXT>(A, K, blockIdx.x, blockIdx.y, smem_raw);
  launch_next();
}

// FP64 and double-float: the edge-parallel tile, with a register budget per kernel variant.
// 56 registers (36 warps per SM) run best or within 3 % of it nearly everywhere measured; the
// FP64 path offers two more to the tuner.
constexpr int edge_regs(int variant) { return variant == 0 ? 56 : (variant == 1 ? 72 : 96); }
template <typename R, int NG, int FLUX, int RECON, int REGS, bool SPLIT>
__global__ void __maxnreg__(REGS) edge_kernel(const StageArgs A, const FluxConsts<R> K) {
  wait_previous();
  if (A.active && *A.active == 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  edge_tile<R, NG, FLUX, RECON, SPLIT>(A, K, blockIdx.x, blockIdx.y, smem_raw);
}

// whether a stage needs the EXT kernel (rectilinear grid, energy source, pressure input)
inline bool stage_needs_ext(const StageArgs& A) {
  return A.G.dxc != nullptr || A.src_q != nullptr || A.bc[SIDE_PX] == BC_PRESSURE_INPUT;
}

}  // namespace cato
