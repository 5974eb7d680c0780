// Programmatic dependent launch for the engine's kernels.  The ops of a plan run back to back on
// one stream, each reading what the one before wrote; launched with programmatic stream
// serialisation, the next kernel is scheduled while the previous one drains (its launch and CTA
// set-up overlap the previous kernel's tail) and holds at griddepcontrol.wait until the previous
// grid has completed and its writes are visible.  Every kernel launched this way calls
// dependent_entry() before it touches global memory.
//
// A kernel lets the next one in as its CTAs leave (what their exit does by itself).  Let in at a kernel's
// start, the next one's CTAs took the first SMs that came free, several to an SM, and waited there for the
// last: the 260 CTAs that slice the second operand of the matvec of bond 1001 then ran on some 40 SMs, and
// the matvec took 178 us instead of 142 (bond 512: 65 and 50; an environment of bond 203, complex128:
// 114 and 107).  Only a kernel that is short and whose follower has one CTA an SM lets it in early,
// by dependent_release().
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace ttg
{
  __device__ __forceinline__ void dependent_entry()
  {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
  }

  __device__ __forceinline__ void dependent_release()
  {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  }

  template <typename... Params, typename... Args>
  cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                               Args &&...args)
  {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
  }
} // namespace ttg
