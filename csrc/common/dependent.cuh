// Launches that overlap the end of the kernel before them (programmatic dependent launch).
//
// A kernel launched with launch_dependent() may begin once every CTA of the kernel before it in the stream has called
// release_dependents() (or ended): its launch latency, barrier and TMEM set-up and tensor-map fetches then pass beside that kernel's
// last work, where an ordinary launch leaves 1-2 us of an idle device between two kernels.  us per pass, ordinary / dependent launches: 12
// layers of width 768 over 777 tokens (98 kernels) 934 / 800, a latent-attention layer over two prompts of 2048 174 / 161 and over 32 decoded
// tokens 126 / 117, attention of a prompt of 1777 tokens 36.3 / 34.5, append + paged decode of 16 sequences 135.5 / 132.2.
// Nothing is given up in order: every thread calls wait_for_previous() before it reads or writes global memory, which returns when all
// kernels before have ended and their writes are visible.
//
// Persistent kernels release theirs when the last loads are under way, so that a waiting dependent does not take the place that a
// communication kernel could have beside them; short ones at once.
// Rules: (1) no global access before wait_for_previous() but prefetches into L2, which return nothing (ptx.cuh), and no CTA without it; (2) TMEM is allocated before release_dependents(), so
// that a dependent's allocation never stands before one that the kernel it waits for still has to make; (3) kernels that wait for flags
// which kernels of other streams or GPUs set release nothing early: a waiting dependent would take the room that those kernels need.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace llmctl {

// The pointers are made anew behind the wait: loads through `const __restrict__` parameters count as invariant, and the compiler could move
// them in front of it.
template <typename... P>                         // pointers
__device__ __forceinline__ void wait_for_previous(P&... p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  ((void)([&] { asm volatile("" : "+l"(p)); }()), ...);
}
__device__ __forceinline__ void release_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace llmctl
