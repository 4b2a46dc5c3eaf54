// prt_launch.cuh - launches of a chain of dependent kernels whose blocks may be scheduled
// while the kernel before them still runs (programmatic dependent launch, sm_90 and later).
//
// A build is a chain of 40 to 50 launches, many of a few microseconds; each used to wait
// for the last block of the one before it, its memory flush and a scheduling gap, 1.5 us in
// all.  With the next kernel's blocks already in place (same GPU, one call in turn with
// ordinary launches): 65,790 triangles 566 -> 502 us, 1,048,576 triangles 1647 -> 1572.  In a
// captured graph the gaps are short already and the edge costs more than it gives (batch
// of 4.6M triangles: 10.19 -> 10.23 ms), so captured builds launch as usual.
//
// Rules for a kernel launched with launch_after:
//  - chain_enter() is its first statement, before any access to global memory: it lets the
//    next kernel of the chain be scheduled (all blocks of this one hold their places by
//    then, so nothing waits for a place that a waiting block holds), then waits until the
//    kernel before it has ended and its writes are visible.  A kernel ends only after that
//    wait, so everything earlier in the stream has ended too.
//  - What an earlier kernel of the chain wrote is read by plain loads, never through the
//    read-only path (__ldg or const __restrict__): such loads need not stay behind the wait.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace prt {

__device__ __forceinline__ void chain_enter() {
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	asm volatile("griddepcontrol.wait;" ::: "memory");
}

// early false: an ordinary launch, after which chain_enter() returns at once.
// A failed launch is left to the caller's next look at cudaGetLastError, as with <<<>>>.
template <typename... P, typename... A>
inline void launch_after(bool early, void (*kernel)(P...), unsigned grid, unsigned block,
                         cudaStream_t st, A... args) {
	cudaLaunchAttribute attr;
	attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr.val.programmaticStreamSerializationAllowed = 1;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(grid);
	cfg.blockDim = dim3(block);
	cfg.stream = st;
	cfg.attrs = &attr;
	cfg.numAttrs = early ? 1 : 0;
	(void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

} // namespace prt
