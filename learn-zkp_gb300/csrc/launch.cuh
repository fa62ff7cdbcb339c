// Dependent launches.  The kernels of one proof form a chain on a stream, most
// of them a few microseconds long, so the time between one kernel's end and the
// next one's first instruction counts.  With programmatic dependent launch the
// next grid is placed while its predecessor still runs and only its first
// memory access waits.  The rules, on which each kernel here relies for the others:
//  * Every block of a kernel launched with launch_chained calls chain_wait(), which
//    waits for the predecessor and only then lets the successor be placed.  So when a
//    block of a grid runs, every block of its predecessor has waited: all
//    launches before the predecessor have completed.
//  * A kernel touches memory that another kernel writes or reads after chain_wait(),
//  * but for the early readers: open_round_kernel, open_tail_kernel,
//    sumcheck_round_kernel, sumcheck_tail_kernel, bb_transcript_round_kernel and
//    bb_tail_kernel load, before it, what a launch before their predecessor wrote (past
//    L1, __ldcg; tables made before the rounds began plainly).  They do so only where the
//    predecessor is a launch of the same chain, made with launch_chained, that does not
//    write what they load: a tree's last launch (which launch_tree makes whenever it is
//    given a root_out) or a fix; in the first round, or where the data came over
//    another stream, they wait first.  They write nothing before it.
// Measured on GB300:
// the 41 launches of a product sumcheck at 2^20 529 -> 388 us, a proof at 2^16
// 1,336 -> 1,273 us.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace bf {

// Returns when the preceding grid of the stream has completed and its writes
// are visible; then the next one may be placed (it waits here in turn).
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t shared, cudaStream_t st,
                                  A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = shared;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
  // reported here: left as the thread's last error, it would fail the next launch that reads that
  if (e != cudaSuccess) (void)cudaGetLastError();
  return e;
}

}  // namespace bf
