// cato_batch.cuh -- many independent grid instances of uneven sizes advanced together: one
// persistent launch per RK stage (and per flux/reconstruction group) walks a work list of
// (instance, tile) items through a device-side queue, so 256 grids cost the launches of one.
// Every instance keeps its own dt, time, iteration and stop condition in a device descriptor,
// so a chunk of steps needs no host round trip and can be captured in a CUDA graph.
#pragma once

#include "cato_ctl.cuh"
#include "cato_stage.cuh"

namespace cato {

struct InstDesc {
  StepCtl ctl;             // per-instance step control (dt, time, iteration, stop, status)
  int ni, nj, pitch, ng;
  int bc[4];
  int limiter, rows_per_cta, flux, recon;
  int raw_pending;         // the first stage uses the uploaded primitives as is
  int prec;                // 0 FP64, 1 mixed, 2 mixed_df (one FP64 layout for all)
  int in_use;
  double gamma, cfl, bc_p;
  Geom G;
  FluxConsts<double> K64;
  FluxConsts<float> K32;
  FluxConsts<df> Kdf;
  double* U[4];            // U^n
  double* S[2][4];         // stage buffers
  double* prim_raw[4];
};

struct BatchStageArgs {
  InstDesc* descs;
  const int4* items;       // (instance, tile x, tile y, rows per tile)
  int n_items;
  int* counter;            // work-queue head, zeroed by batch_step_begin
  int stage, kind, last;
  double a, b, coef;
};

// Build one instance's StageArgs for this stage: the device-side twin of the single-instance
// host sequencing (cato_capi.cu enqueue_step).
template <typename R>
__device__ __forceinline__ void batch_stage_args(InstDesc* d, const BatchStageArgs& B,
                                                 StageArgs& A) {
  A.ni = d->ni;
  A.nj = d->nj;
  A.pitch = d->pitch;
#pragma unroll
  for (int k = 0; k < 4; ++k) A.bc[k] = d->bc[k];
  A.limiter = d->limiter;
  A.rows_per_cta = d->rows_per_cta;
  A.kind = B.kind;
  A.last = B.last;
  A.a = B.a;
  A.b = B.b;
  A.coef = B.coef;
  A.dt = &d->ctl.dt;
  A.active = nullptr;
  A.dt_min = &d->ctl.dt_min;
  A.status = &d->ctl.status;
  A.gamma = d->gamma;
  A.bc_p = d->bc_p;
  A.G = d->G;
  // single-handle features the batch does not carry (configurations are rejected at add)
  A.pbc_edge = nullptr;
  A.pbc_ng = 0;
  A.src_q = nullptr;
  const bool raw = (B.stage == 0) && d->raw_pending;
  double* const* prev = (B.stage == 0) ? d->U : d->S[(B.stage - 1) & 1];
  double* const* out = B.last ? d->U : d->S[B.stage & 1];
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    A.Uk[v] = prev[v];
    A.Ua[v] = d->U[v];
    A.Uo[v] = out[v];
    A.Pin[v] = raw ? d->prim_raw[v] : nullptr;
  }
}

// The persistent loop of a batch kernel: every CTA pulls (instance, tile) items from the queue and
// hands them to tile(A, descriptor, tile x, tile y).  SHARED: the tile's arguments are built once, in
// shared memory; as each thread's own, indexed by variable, they lay in local memory, whose 688
// bytes a thread are 120 MB of the L2 with an edge kernel's 36 warps on every SM (48 random-circle
// grids, FP64 SLAU + MLP5: 1.93 GB written to DRAM per stage for 0.13 GB of results).
template <typename R, bool SHARED, typename Tile>
__device__ __forceinline__ void batch_loop(const BatchStageArgs& B, Tile tile) {
  wait_previous();
  __shared__ int s_item;
  __shared__ __align__(16) unsigned char s_args[SHARED ? sizeof(StageArgs) : 16];
  const bool first = threadIdx.x == 0 && threadIdx.y == 0;
  auto fill = [&](StageArgs& A, int it) {
    const int4 w = B.items[it];
    batch_stage_args<R>(B.descs + w.x, B, A);
    A.rows_per_cta = w.w;
    A.block = 4;  // batch_shape
  };
  for (;;) {
    __syncthreads();  // the previous tile is done with shared memory and s_item
    if (first) {
      const int it = atomicAdd(B.counter, 1);
      s_item = it;
      if (SHARED && it < B.n_items) fill(*reinterpret_cast<StageArgs*>(s_args), it);
    }
    __syncthreads();
    const int it = s_item;
    if (it >= B.n_items) break;
    const int4 w = B.items[it];
    InstDesc* d = B.descs + w.x;
    if (!d->ctl.active) continue;
    if constexpr (SHARED) {
      tile(*reinterpret_cast<const StageArgs*>(s_args), d, w.y, w.z);
    } else {
      StageArgs A;
      fill(A, it);
      tile(A, d, w.y, w.z);
    }
  }
}

// FP32; no rectilinear grid, source or pressure input in a batch: the lean tile
template <int NG, int FLUX, int RECON>
__global__ void __maxnreg__(f32_batch_regs(FLUX, RECON))
    batch_stage_kernel(const BatchStageArgs B) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  batch_loop<float, false>(B, [&](const StageArgs& A, const InstDesc* d, int bx, int by) {
    tile_of<NG, FLUX, RECON, false, batch_tvd_tile_of(FLUX, RECON)>(A, d->K32, bx, by, smem_raw);
  });
}

// FP64 and double-float
template <typename R, int NG, int FLUX, int RECON>
__global__ void __maxnreg__(edge_regs(0)) batch_edge_kernel(const BatchStageArgs B) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  batch_loop<R, true>(B, [&](const StageArgs& A, const InstDesc* d, int bx, int by) {
    if constexpr (Prec<R>::kind == 0) edge_tile<R, NG, FLUX, RECON, false>(A, d->K64, bx, by, smem_raw);
    else edge_tile<R, NG, FLUX, RECON, false>(A, d->Kdf, bx, by, smem_raw);
  });
}

}  // namespace cato
