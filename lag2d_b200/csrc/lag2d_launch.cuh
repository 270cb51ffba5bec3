// Programmatic dependent launch of the passes on a step's main chain: a pass comes
// up while the one before it runs, and reads ahead what that one does not write.
//
// Order.  A pass calls await_previous once, before it first reads or overwrites
// anything that the pass before it (or a side pass that joins there) works on, and
// only then lets the next one up.  So by the time a pass starts, all passes but the
// last before it are complete: what those wrote may be read ahead of the wait, what
// the last one writes may not, and nothing may be written ahead of it.
#pragma once
#include <cuda_runtime.h>

namespace lag2d {

// the results of the kernel this one was launched behind are there (at once in a
// plain launch); the kernel launched behind this one may come up
__device__ __forceinline__ void await_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Meshes of up to this many cells use it.  us a step without / with: P2 16 x 16
// 71 / 64, 64 x 64 78 / 71, 128 x 128 102 / 92, 256 x 256 205 / 194, Sedov
// 128 x 128 149 / 139, RZ 100 x 100 47 / 42; with the integrals that need no u* ahead
// of the wait 63, 68, 88, 194, 138, 40.  On a mesh that
// fills the chip many times the waiting blocks take room from the side passes
// (1024 x 1024 2501 / 2555).
constexpr int kBehindMax = 131072;

// behind = 0: a plain launch
template <typename... P, typename... A>
void launch_behind(bool behind, void (*k)(P...), int grid, int block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &a;
  c.numAttrs = behind ? 1 : 0;
  cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);
}

}  // namespace lag2d
