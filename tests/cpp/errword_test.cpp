// Unit test of the host side of an error word (prt_errword.h): a word without bits is not
// written, and bits set by several threads while another takes them are each taken once.
#include <sys/mman.h>
#include <unistd.h>

#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

#include "prt_errword.h"

int main() {
	// A page that may only be read: a write would end the process.
	const long page = sysconf(_SC_PAGESIZE);
	void *p = mmap(nullptr, (size_t)page, PROT_READ, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
	if (p == MAP_FAILED || prt::take_error_bits(static_cast<uint32_t *>(p)) != 0u) {
		std::printf("FAILED empty word\n");
		return 1;
	}
	uint32_t word = 0;
	constexpr int kThreads = 4, kSets = 20000;
	std::atomic<int> running{kThreads};
	long set[kThreads] = {}, taken[kThreads] = {};
	std::vector<std::thread> threads;
	for (int k = 0; k < kThreads; ++k)
		threads.emplace_back([&, k] {
			for (int i = 0; i < kSets; ++i)
				set[k] += !(__atomic_fetch_or(&word, 1u << k, __ATOMIC_ACQ_REL) & (1u << k));
			--running;
		});
	for (bool last = false; !last;) {
		last = running == 0;
		const uint32_t bits = prt::take_error_bits(&word);
		for (int k = 0; k < kThreads; ++k)
			taken[k] += (bits >> k) & 1u;
	}
	for (auto &t : threads)
		t.join();
	for (int k = 0; k < kThreads; ++k)
		if (set[k] != taken[k]) {
			std::printf("FAILED bit %d: set %ld times, taken %ld\n", k, set[k], taken[k]);
			return 1;
		}
	std::printf("OK\n");
	return 0;
}
