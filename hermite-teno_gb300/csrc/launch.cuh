// Programmatic dependent launch: a kernel's blocks may become resident, and set up what does not depend
// on earlier kernels, while the kernel before it in the stream still runs.  Every kernel launched by
// launch_early calls grid_wait before it touches global memory that an earlier kernel writes, or reads
// before this one writes it.  grid_release lets the next such kernel start; its blocks come after all of
// this kernel's have started, so nothing that runs waits for them.
#pragma once

#include <cuda_runtime.h>

namespace hteno {

// Until the previous kernel of the stream has completed and its writes are visible (at once if this one
// was launched without the attribute).
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// grid_wait keeps plain loads below it, but not those that count as loads of memory that nobody else
// writes: by __ldg or through a const __restrict__ parameter (which may also take the path that is not kept
// coherent), and through any other __restrict__ parameter.  A kernel launched early reads what an earlier
// kernel writes by plain loads through pointers that are not __restrict__, by load_behind, or through a
// pointer that the compiler knows only from here on, after_wait(p), behind grid_wait.
template <typename T>
__device__ __forceinline__ T* after_wait(T* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}
// A plain load that the compiler keeps where it stands.  (The halo of an FV 2D tile by ordinary loads: 123
// instead of 96 registers in the batch kernel, batches of small grids 1120 -> 1400 us per ten steps.)
__device__ __forceinline__ double load_behind(const double* p) {
  double r;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(r) : "l"(__cvta_generic_to_global(p)));
  return r;
}

// kernel<<<grid, block, smem, st>>>(args...), early or (a stream under capture, timed launches) not.
template <typename... P, typename... A>
inline cudaError_t launch_early(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                const A&... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

}  // namespace hteno
