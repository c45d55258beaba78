// Programmatic dependent launch for the library's kernel chains (sm_103a).
//
// A step is a chain of short kernels, and on small grids the gap between one kernel's
// last store and the next one's first instruction (drain, launch, block setup) is as long
// as the kernels. With programmatic stream serialization the next kernel's blocks are
// placed while the previous one still runs and wait at pdl_begin() until it has finished
// and its stores are visible. Every kernel launched through pdl_launch calls pdl_begin()
// before it touches global memory: the wait covers all earlier work of the stream, since
// a kernel cannot finish before its own wait has passed. The trigger follows the wait, so
// at most one kernel's blocks are parked behind a running one, and they are placed only
// when every block of the running kernel has started (they never take a slot from it).
//
// Measured per step or call with and without it: 2D 256^2 70.3 -> 53.8 us, 128^2 x 8
// 70.9 -> 57.6 us, 3D 64^3 107 -> 89 us, 128^3 with ekin_tot and u 393 -> 343 us, NUFFT
// update of 32^3 particles 98 -> 80 us, two steps and their adjoint at 128^3 2.40 -> 2.15 ms;
// 256^3 and 512^3 steps, whose kernels run for 40 to 1300 us, stay within 0.4%.
#pragma once

#include <cuda_runtime.h>

namespace l3es {

__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// SMs of the current device (GB300: 152), for the rules that compare a launch's blocks with
// them; 0 if the device cannot tell.
inline int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    cudaGetLastError();
  return sms;
}

template <typename... P, typename... A>
inline void pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace l3es
