// prt_errword.h - a word of error bits that kernels set and the host takes.
//
// A context's word is pinned host memory (prt_b200_ctx::h_err).  The host takes it after it has
// waited for its own work, while kernels that other threads queued on other streams may still
// run and set bits, so both sides' accesses are atomic with respect to each other: the
// kernels' at system scope (the host link is coherent and carries atomics), the host's an
// atomic exchange.  Nothing here clears a bit that its caller has not looked at.
#pragma once

#include <stdint.h>

namespace prt {

// Host: the bits set since they were last taken.  A word without any is only read.
inline uint32_t take_error_bits(uint32_t *word) {
	if (__atomic_load_n(word, __ATOMIC_ACQUIRE) == 0u)
		return 0u;
	return __atomic_exchange_n(word, 0u, __ATOMIC_ACQ_REL);
}

#ifdef __CUDACC__
__device__ __forceinline__ void set_error_bits(uint32_t *word, uint32_t bits) {
	atomicOr_system(word, bits);
}
__device__ __forceinline__ void clear_error_bits(uint32_t *word, uint32_t bits) {
	atomicAnd_system(word, ~bits);
}
#endif

} // namespace prt
