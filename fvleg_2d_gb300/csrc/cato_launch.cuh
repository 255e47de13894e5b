// cato_launch.cuh -- host-side launchers of the stage kernels, instantiated per (precision, flux)
// in separate translation units (stage_inst.cu compiled once per pair) so that the FP64 ones can
// be built with --fmad=false and the build parallelises.
#pragma once

#include <algorithm>
#include <atomic>

#include "cato_batch.cuh"
#include "cato_shape.h"
#include "cato_stage.cuh"

namespace cato {

// A kernel's function attributes (here its dynamic shared-memory limit) belong to the GPU that
// is current when they are set, so the "already set" flags are kept per device.
constexpr int kMaxDevices = 64;
struct PerDevice {
  std::atomic<bool> done[kMaxDevices] = {};
  std::atomic<int> sms[kMaxDevices] = {};
};
// the current device, or -1 when it cannot be read or lies beyond kMaxDevices
inline int launch_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
  return dev;
}

// SMs of the current device (1 when it cannot be read)
inline int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    (void)cudaGetLastError();
  return n > 0 ? n : 1;
}

// Raises kernel's dynamic shared-memory limit once per device.
template <typename F>
inline cudaError_t allow_smem(PerDevice& attr, int dev, F* kernel, size_t bytes) {
  if (attr.done[dev].load(std::memory_order_acquire)) return cudaSuccess;
  const cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  int n = 0;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  attr.sms[dev].store(n > 0 ? n : 1);
  attr.done[dev].store(true, std::memory_order_release);
  return cudaSuccess;
}
// the largest shared memory an edge-parallel kernel may be launched with
template <typename R> inline size_t edge_smem_limit(int ng) {
  return std::max({edge_smem_bytes<R>({64, 4, 9}, ng), edge_smem_bytes<R>({128, 2, 5}, ng),
                   edge_smem_bytes<R>({32, 2, 10}, ng)});
}
inline bool edge_shape_ok(EdgeShape s) {
  return s.columns >= 32 && s.columns <= 128 && s.columns % 32 == 0 && s.block >= 1 &&
         s.block * s.columns <= 256 && s.warps >= 2 * s.block + 1 &&
         s.columns * s.warps <= kEdgeThreads;
}

template <int NG, int FLUX, int RECON, bool EXT>
cudaError_t launch_strip(const StageShape& s, bool warm, cudaStream_t stream, const StageArgs& A,
                         const FluxConsts<float>& K) {
  static PerDevice attr;
  constexpr bool TVD = tvd_tile_of(FLUX, RECON);
  const int dev = launch_device();
  if (dev < 0) return cudaErrorInvalidDevice;
  cudaError_t e = allow_smem(attr, dev, stage_kernel<NG, FLUX, RECON, EXT>,
                             tile_smem_bytes(256, NG, FLUX, TVD));
  if (e != cudaSuccess || warm) return e;
  const int W = s.threads - 2 * NG;
  const dim3 grid((A.ni + W - 1) / W, (A.nj + s.rows - 1) / s.rows);
  return launch_overlapped(stage_kernel<NG, FLUX, RECON, EXT>, grid, dim3(s.threads),
                           tile_smem_bytes(s.threads, NG, FLUX, TVD), stream, A, K);
}

template <typename R, int NG, int FLUX, int RECON, int REGS, bool SPLIT = false>
cudaError_t launch_edge(const StageShape& s, bool warm, cudaStream_t stream, const StageArgs& A,
                        const FluxConsts<R>& K) {
  static PerDevice attr;
  const int dev = launch_device();
  if (dev < 0) return cudaErrorInvalidDevice;
  cudaError_t e = allow_smem(attr, dev, edge_kernel<R, NG, FLUX, RECON, REGS, SPLIT>,
                             edge_smem_limit<R>(NG));
  if (e != cudaSuccess || warm) return e;
  EdgeShape es{s.threads, s.block, s.warps};
  // the CTA's warps fit the register file: a quarter of them in each of its four 16 Ki parts
  es.warps = std::min(es.warps, 4 * (16384 / (32 * REGS)) * 32 / es.columns);
  es.block = std::min(es.block, (es.warps - 1) / 2);
  if (!SPLIT) es.warps = 2 * es.block + 1;
  if (!edge_shape_ok(es) || es.split() != SPLIT) return cudaErrorInvalidValue;
  const int W = es.columns - 2 * NG;
  const dim3 grid((A.ni + W - 1) / W, (A.nj + s.rows - 1) / s.rows);
  StageArgs B = A;
  B.block = es.block;
  return launch_overlapped(edge_kernel<R, NG, FLUX, RECON, REGS, SPLIT>, grid,
                           dim3(es.columns, es.warps), edge_smem_bytes<R>(es, NG), stream, B, K);
}

// One stage of one grid; warm: only prepare every kernel of the scheme (outside stream captures).
// The FP32 path has a lean variant without the rectilinear, source and pressure-input code (it is
// issue-bound: those checks cost ~3 %).  The FP64 path has one kernel per register budget
// (edge_regs).
template <typename R, int NG, int FLUX, int RECON>
cudaError_t launch_stage_one(const StageShape& s, bool warm, cudaStream_t stream,
                             const StageArgs& A, const FluxConsts<R>& K) {
  if constexpr (Prec<R>::kind == 1) {
    if (warm) {
      cudaError_t e = launch_strip<NG, FLUX, RECON, false>(s, true, stream, A, K);
      if (e != cudaSuccess) return e;
    } else if (!stage_needs_ext(A)) {
      return launch_strip<NG, FLUX, RECON, false>(s, false, stream, A, K);
    }
    return launch_strip<NG, FLUX, RECON, true>(s, warm, stream, A, K);
  } else {
    const StageForm form = stage_form(s, Prec<R>::kind == 0 ? CATO_FP64 : CATO_MIXED_DF);
    if (warm) {
      cudaError_t e = launch_edge<R, NG, FLUX, RECON, edge_regs(0), true>(s, true, stream, A, K);
      if (e != cudaSuccess) return e;
    } else if (form.split) {
      return launch_edge<R, NG, FLUX, RECON, edge_regs(0), true>(s, false, stream, A, K);
    }
    if constexpr (Prec<R>::kind == 0) {
      if (warm) {
        cudaError_t e = launch_edge<R, NG, FLUX, RECON, edge_regs(1)>(s, true, stream, A, K);
        if (e == cudaSuccess)
          e = launch_edge<R, NG, FLUX, RECON, edge_regs(2)>(s, true, stream, A, K);
        if (e != cudaSuccess) return e;
      } else if (form.variant == 1) {
        return launch_edge<R, NG, FLUX, RECON, edge_regs(1)>(s, false, stream, A, K);
      } else if (form.variant == 2) {
        return launch_edge<R, NG, FLUX, RECON, edge_regs(2)>(s, false, stream, A, K);
      }
    }
    return launch_edge<R, NG, FLUX, RECON, edge_regs(0)>(s, warm, stream, A, K);
  }
}

// recon: 0 = TVD2 (minmod / superbee / van Leer), 3 = MLP3, 5 = MLP5
template <typename R, int FLUX>
inline cudaError_t launch_stage_flux(int recon, const StageShape& s, bool warm,
                                     cudaStream_t stream, const StageArgs& A,
                                     const FluxConsts<R>& K) {
  switch (recon) {
    case 0: return launch_stage_one<R, 2, FLUX, 0>(s, warm, stream, A, K);
    case 3: return launch_stage_one<R, 2, FLUX, 3>(s, warm, stream, A, K);
    case 5: return launch_stage_one<R, 3, FLUX, 5>(s, warm, stream, A, K);
    default: return cudaErrorInvalidValue;
  }
}

// The shape of a batch launch for a plan's CTA width: FP32 strips are as wide as the plan says;
// the edge-parallel tiles half as wide (32 to 64 columns), in blocks of 4 rows.
template <typename R> inline EdgeShape batch_shape(int threads) {
  if (Prec<R>::kind == 1) return {threads, 0, 0};
  return {threads < 128 ? 32 : 64, 4, 9};
}

// Persistent batch launch: as many CTAs as can be resident, each looping over work items.
template <typename R, int NG, int FLUX, int RECON>
cudaError_t launch_batch_one(int threads, cudaStream_t stream, const BatchStageArgs& B) {
  static PerDevice attr;
  const int dev = launch_device();
  if (dev < 0) return cudaErrorInvalidDevice;
  const EdgeShape shape = batch_shape<R>(threads);
  void (*kernel)(const BatchStageArgs);
  size_t smem, most;
  dim3 block;
  if constexpr (Prec<R>::kind == 1) {
    kernel = batch_stage_kernel<NG, FLUX, RECON>;
    smem = tile_smem_bytes(threads, NG, FLUX, batch_tvd_tile_of(FLUX, RECON));
    most = tile_smem_bytes(256, NG, FLUX, batch_tvd_tile_of(FLUX, RECON));
    block = dim3(threads);
  } else {
    kernel = batch_edge_kernel<R, NG, FLUX, RECON>;
    smem = edge_smem_bytes<R>(shape, NG);
    most = edge_smem_limit<R>(NG);
    block = dim3(shape.columns, shape.warps);
  }
  cudaError_t e = allow_smem(attr, dev, kernel, most);
  if (e != cudaSuccess) return e;
  if (B.n_items <= 0) return cudaSuccess;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, (int)(block.x * block.y), smem);
  if (e != cudaSuccess) return e;
  long long grid = (long long)(per_sm > 0 ? per_sm : 1) * attr.sms[dev].load();
  if (grid > B.n_items) grid = B.n_items;
  return launch_overlapped(kernel, dim3((unsigned)grid), block, smem, stream, B);
}

template <typename R, int FLUX>
inline cudaError_t launch_batch_flux(int recon, int threads, cudaStream_t stream,
                                     const BatchStageArgs& B) {
  switch (recon) {
    case 0: return launch_batch_one<R, 2, FLUX, 0>(threads, stream, B);
    case 3: return launch_batch_one<R, 2, FLUX, 3>(threads, stream, B);
    case 5: return launch_batch_one<R, 3, FLUX, 5>(threads, stream, B);
    default: return cudaErrorInvalidValue;
  }
}

// Every (precision, NG, flux, reconstruction) kernel is instantiated in exactly one translation
// unit (stage_inst.cu, compiled once per precision and flux, and for the slow double-float units
// once per reconstruction and kernel kind); everywhere else these are extern.
#define CATO_DECLARE_ONE(R, F, NG, RC)                                                         \
  extern template cudaError_t launch_stage_one<R, NG, F, RC>(const StageShape&, bool,          \
                                                             cudaStream_t, const StageArgs&,   \
                                                             const FluxConsts<R>&);            \
  extern template cudaError_t launch_batch_one<R, NG, F, RC>(int, cudaStream_t,               \
                                                             const BatchStageArgs&);
#define CATO_DECLARE_STAGE(R, F) \
  CATO_DECLARE_ONE(R, F, 2, 0) CATO_DECLARE_ONE(R, F, 2, 3) CATO_DECLARE_ONE(R, F, 3, 5)
#define CATO_DECLARE_PREC(R)                                                      \
  CATO_DECLARE_STAGE(R, 0) CATO_DECLARE_STAGE(R, 1) CATO_DECLARE_STAGE(R, 2)      \
  CATO_DECLARE_STAGE(R, 3) CATO_DECLARE_STAGE(R, 4) CATO_DECLARE_STAGE(R, 5)      \
  CATO_DECLARE_STAGE(R, 6) CATO_DECLARE_STAGE(R, 7) CATO_DECLARE_STAGE(R, 8)
CATO_DECLARE_PREC(double)
CATO_DECLARE_PREC(float)
CATO_DECLARE_PREC(df)
#undef CATO_DECLARE_PREC
#undef CATO_DECLARE_STAGE
#undef CATO_DECLARE_ONE

template <typename R>
inline cudaError_t launch_stage(int flux, int recon, const StageShape& h, bool warm, cudaStream_t s,
                                const StageArgs& A, const FluxConsts<R>& K) {
  switch (flux) {
    case 0: return launch_stage_flux<R, 0>(recon, h, warm, s, A, K);
    case 1: return launch_stage_flux<R, 1>(recon, h, warm, s, A, K);
    case 2: return launch_stage_flux<R, 2>(recon, h, warm, s, A, K);
    case 3: return launch_stage_flux<R, 3>(recon, h, warm, s, A, K);
    case 4: return launch_stage_flux<R, 4>(recon, h, warm, s, A, K);
    case 5: return launch_stage_flux<R, 5>(recon, h, warm, s, A, K);
    case 6: return launch_stage_flux<R, 6>(recon, h, warm, s, A, K);
    case 7: return launch_stage_flux<R, 7>(recon, h, warm, s, A, K);
    case 8: return launch_stage_flux<R, 8>(recon, h, warm, s, A, K);
    default: return cudaErrorInvalidValue;
  }
}

template <typename R>
inline cudaError_t launch_batch(int flux, int recon, int threads, cudaStream_t s,
                                const BatchStageArgs& B) {
  switch (flux) {
    case 0: return launch_batch_flux<R, 0>(recon, threads, s, B);
    case 1: return launch_batch_flux<R, 1>(recon, threads, s, B);
    case 2: return launch_batch_flux<R, 2>(recon, threads, s, B);
    case 3: return launch_batch_flux<R, 3>(recon, threads, s, B);
    case 4: return launch_batch_flux<R, 4>(recon, threads, s, B);
    case 5: return launch_batch_flux<R, 5>(recon, threads, s, B);
    case 6: return launch_batch_flux<R, 6>(recon, threads, s, B);
    case 7: return launch_batch_flux<R, 7>(recon, threads, s, B);
    case 8: return launch_batch_flux<R, 8>(recon, threads, s, B);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace cato
