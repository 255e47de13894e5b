// cato_ctl.cuh -- device-resident step control shared by the single-instance and batch paths.
#pragma once

#include <cuda_runtime.h>

namespace cato {

// Device-resident step control: lets a chunk of steps run (and be captured in a CUDA graph)
// without host round trips.  `active` gates every kernel of a step.
struct StepCtl {
  double dt;          // dt of the current step
  double time;        // simulation time after the last active step
  double t_end;       // stop once time >= t_end (main.f90:138)
  double fixed_dt;    // > 0: use this dt instead of the CFL dt (use_constant_delta_t)
  long long iter;     // iteration counter
  long long max_iter; // stop once iter >= max_iter
  unsigned long long dt_min;  // CFL dt of the current state (bits; ~0 = none)
  int active;
  int status;         // ST_* bits of the current state
  double t_create;    // time the state was created at (upload / set_time): the flux solver of
                      // the persistent fluid keeps it under rk(m,n) (pressure-input table time)
  double t_step;      // time at the start of the current step (energy source term time)
};

// Programmatic dependent launch: a kernel of a step is set up while its predecessor drains and
// waits here, before its first access to memory, until the predecessor's results are complete.
// Its blocks start when all of the predecessor's have passed launch_next or ended.  The FP32
// kernel of a single grid calls it after its tile; the edge-parallel kernels do not: blocks that
// start while others still run are placed unevenly, and a grid of about one block per SM then has
// two on some (FP64 400 x 40: 54.0 us a step without the call, 62.3 with it, 62.0 with plain
// launches; FP32 64 x 48: 17.9 us with it, 28.7 with plain launches).  Nor do the persistent batch
// kernels: from within a tile the call would let the next stage's blocks wait on the SMs while the
// queue still has items (served mix 131.0 us a step without it, 130.6 with it after the first
// tile).  No-ops in a plain launch.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void launch_next() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// What the predecessor wrote is read with this or a plain load: the read-only path (__ldg) is for
// data that nothing writes from the kernel's start on, and the wait does not order it.  A plain load
// of the stage state, whose address the compiler does not know to be global, costs FP32 up to 18 %
// (HLLC 4096^2: 1398 us a step, 1258 with this as with __ldg; AUSMPW+ 2048^2: 414, 350).
__device__ __forceinline__ double load_global(const double* p) {
  double x;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(x) : "l"(__cvta_generic_to_global(p)));
  return x;
}
// Launches kernel(args...) so that it may start while the stream's previous kernel drains.
template <typename... P, typename... A>
inline cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                                     cudaStream_t stream, const A&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

__device__ __forceinline__ double decode_dt(unsigned long long b) {
  return b == ~0ULL ? INFINITY : __longlong_as_double((long long)b);
}

}  // namespace cato
