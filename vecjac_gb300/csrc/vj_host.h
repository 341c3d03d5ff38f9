// Host-side services shared by the entry points: device discovery, a growable device
// staging buffer for the host-pointer forms, and a pair of library-owned streams.
#pragma once
#include <mutex>
#include <cfenv>
#include <cstddef>
#include <cuda_runtime.h>

#include "../../include/vecjac_gb300.h"

namespace vj {
namespace host {

// Round-to-nearest for the host-side arithmetic of one call (tolerances, rescaling
// bounds), whatever rounding mode the caller's thread has; the caller's mode is restored.
struct NearestRounding {
  int saved;
  NearestRounding() : saved(fegetround())
  {
    if (saved != FE_TONEAREST)
      fesetround(FE_TONEAREST);
  }
  ~NearestRounding()
  {
    if (saved != FE_TONEAREST)
      fesetround(saved);
  }
  NearestRounding(const NearestRounding &) = delete;
  NearestRounding &operator=(const NearestRounding &) = delete;
};

// true when a CUDA device is usable (checked once; the current device is used)
bool gpu_ready();
// Library state is kept per device (the current device of each call): SM count, staging
// buffers, streams, the batch queues.
constexpr int MAX_DEVICES = 64;
int device_slot();
int sm_count();
// the device can read and write pageable host memory (and VJ_STAGED is not set)
bool pageable_access();
// p (NULL counts as true) is page-locked host memory (cudaHostAlloc / cudaHostRegister)
bool host_pinned(const void *p);
// p is memory that this thread may write (not NULL, not device memory)
bool host_written(const void *p);

// device memory reused across host-API calls; grows on demand, never shrinks
struct Staging {
  char *ptr = nullptr;
  size_t size = 0;
  bool reserve(size_t bytes);
};
Staging &staging();
Staging &staging2();
// scratch of the mixed-precision SVD (its inner SVD calls use staging2)
Staging &staging3();

// page-locked host memory for the outputs of one small 2x2 call (SMALL_OUT bytes of arrays and
// their permutation words), allocated on first use, one per device, under host_call_lock
constexpr size_t SMALL_OUT = (size_t)512 << 10;
char *small_out();

// Device memory for one call of the batched SVD (always the same size): its work queues and
// what its CTAs need to know of the batch. take before the call's launches, done after them, on
// the same stream. No two calls that may run at the same time share it: a call enqueued to
// run has a slot that waits for the call before on it, a captured one a slot of the graph's own,
// given back when the graph and its instances are gone.
struct BatchPlanSlot {
  char *ptr = nullptr;
  int slot = -1;  // >= 0: an event is to be recorded
};
bool batch_plan_take(size_t bytes, cudaStream_t s, BatchPlanSlot &p);
bool batch_plan_done(const BatchPlanSlot &p, cudaStream_t s);

// two non-blocking streams owned by the library
bool streams2(cudaStream_t s[2]);

// Taken by the host-pointer entry points (dbjac2_ ... zsplit_ ...), which share the
// device's staging buffers: calls from several host threads run one at a time on a device,
// so those entry points are reentrant like the reference's. (Recursive: a host form may
// call another.)
std::recursive_mutex &host_call_lock();

// launch with programmatic stream serialisation (the kernel calls pdl_enter first)
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

// per-sweep statistics of the last SVD (transformed pairs per sweep)
void trace_reset();
void trace_sweep(unsigned sweep, unsigned long long rotations);
// per-phase cycle counts (VJ_TRACE=1 in the environment enables their collection)
bool trace_enabled();
void trace_phases(const unsigned long long *cycles, int count);

// phase times (ms) of the last mixed-precision SVD, its number of FP32 launches and whether
// its FP32 stages ran as block sweeps on the tensor cores (1) or by small blocks or pairs (0)
void mixed_phases_set(double fp32, double gemm, double fp64, double fin, double fp32_steps, double block);

// elements per chunk of a host-pointer 2x2 call (a multiple of `lanes`)
long long bjac2_chunk(long long n, size_t elem, bool cplx, int lanes);

}  // namespace host
}  // namespace vj
