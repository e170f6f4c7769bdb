// Launches of kernels that follow one another on a stream.
//
// A small step is bound by the gaps between its kernels: a plain launch starts
// only once the kernel before it has completed and been flushed.  chain()
// launches with programmatic stream serialization, so that the launch itself
// is over by then and the blocks only wait (chain_wait).  One step of 16k
// Gaussians at 256x256, 18 kernels: 302 -> 256 us; a 611x397 render of 20k, 14
// kernels: 204 -> 178.  Letting the next kernel's blocks in as soon as all of
// this one's have started (griddepcontrol.launch_dependents) takes 272 and 187:
// they hold registers and shared memory that the running kernel's blocks use.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

namespace sky {

// The first statement of every kernel that chain() launches: waits until the
// kernel before it in the stream has completed and its writes are visible
// (nothing to wait for after a plain launch).  Every block runs it, also those
// with no work: a kernel that completed before its predecessor would let its
// own successor start too early.
// p: every pointer parameter of the kernel.  Loads through a const __restrict__
// parameter are invariant to the compiler, which may move them above a memory
// clobber; passed through an empty volatile statement behind the wait, the
// pointers, and with them the loads, cannot go before it.
template <class... P>
__device__ __forceinline__ void chain_wait(P&... p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  auto behind = [](auto& q) {
    unsigned long long a = reinterpret_cast<unsigned long long>(q);
    asm volatile("" : "+l"(a)::"memory");
    q = reinterpret_cast<std::remove_reference_t<decltype(q)>>(a);
  };
  (behind(p), ...);
}

// programmatic: false launches as <<<>>> does.
template <class... P, class... A>
cudaError_t chain_if(bool programmatic, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                     cudaStream_t s, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = programmatic ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <class... P, class... A>
cudaError_t chain(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  return chain_if(true, kernel, grid, block, smem, s, args...);
}

}  // namespace sky
