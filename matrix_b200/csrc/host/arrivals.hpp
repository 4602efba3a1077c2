// Waiting for results that a kernel writes straight into page-locked memory. The words are canonical residues, so a word of all ones is
// none of them: the host sets them to that before the launch and looks until every one has changed. That sees a pass's sums 3.4 us
// before a stream synchronisation returns (launch, empty kernel and wait: 8.8 against 12.1 us). The kernel may still be on its
// way out then, which the stream's order hides from later work on it; who gives memory to other streams synchronises first, or waits
// for a word that the kernel stores behind everything else, fenced.
// A caller whose device flags ask for yielding or blocking waits gets the synchronisation instead.
// A pass that takes longer than the polls, fails, or gives up one of its own waits (it writes no sums then) ends with a synchronisation.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cstring>
#include "../common.cuh"

namespace mbhost {

constexpr uint64_t NOT_ARRIVED = ~0ULL;
constexpr int ARRIVAL_POLLS = 1 << 15;   // about 1.5 ms

inline void expect_words(uint64_t* p, size_t n) { std::memset(p, 0xFF, n * sizeof(uint64_t)); }

// The caller has asked for waits that leave the core to others (cudaSetDeviceFlags).
inline bool waits_without_spinning() {
    unsigned flags = 0;
    if (cudaGetDeviceFlags(&flags) != cudaSuccess) return false;
    const unsigned how = flags & cudaDeviceScheduleMask;
    return how == cudaDeviceScheduleYield || how == cudaDeviceScheduleBlockingSync;
}
inline int await_words(const uint64_t* p, size_t n) {
    int left = ARRIVAL_POLLS;
    for (size_t i = 0; i < n; i++)
        while (__atomic_load_n(p + i, __ATOMIC_RELAXED) == NOT_ARRIVED) {
            if (left == ARRIVAL_POLLS && waits_without_spinning()) left = 0;   // asked while the pass runs
            if (left-- <= 0) return cudaStreamSynchronize(MB_STREAM) == cudaSuccess ? MB_OK : MB_ERR_CUDA;
#if defined(__x86_64__)
            __builtin_ia32_pause();
#endif
        }
    __atomic_thread_fence(__ATOMIC_ACQUIRE);
    return MB_OK;
}

}  // namespace mbhost
