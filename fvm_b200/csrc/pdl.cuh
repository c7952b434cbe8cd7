// Programmatic dependent launch: a kernel lets the next one of its stream be
// launched early and waits for all before it ahead of its first read of
// anything they write. Every kernel of a chain waits, so a wait covers all
// earlier kernels. Pointers to what the chain writes carry no __restrict__:
// such loads are invariant to the compiler and may be moved above the wait.
#pragma once

#include <cuda_runtime.h>

#define FVM_PDL_TRIGGER() asm volatile("griddepcontrol.launch_dependents;" ::: "memory")
#define FVM_PDL_WAIT() asm volatile("griddepcontrol.wait;" ::: "memory")
#define FVM_PDL()      \
  do {                 \
    FVM_PDL_TRIGGER(); \
    FVM_PDL_WAIT();    \
  } while (0)

namespace fvm {

// kernels and copies that this thread has issued on the paths of a solve
inline thread_local long long launchesIssued = 0;

template <typename... KArgs, typename... Args>
inline void pdl_launch_smem(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                            Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  launchesIssued++;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <typename... KArgs, typename... Args>
inline void pdl_launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t st, Args... args) {
  pdl_launch_smem(kernel, grid, block, 0, st, args...);
}

}  // namespace fvm
