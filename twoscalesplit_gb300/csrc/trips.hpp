// trips.hpp -- how the entries of a list are spread over a kernel's threads (host and
// device code, so that the index arithmetic is tested on the CPU).
#pragma once

#ifdef __CUDACC__
#define TSS_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TSS_HOST_DEVICE inline
#endif

namespace tss {

// f(base) for each trip of thread `thread` of block `block`: the trip's entries are base,
// base + threads, ..., base + (U - 1) threads, those below n (n < 2^31) taken.  Unsigned: a
// trip past the end of a list of nearly 2^31 entries starts above 2^31 and must not wrap
// to a negative index (blocks * threads * U < 2^31).
template <int U, class F>
TSS_HOST_DEVICE void for_trips(unsigned n, unsigned block, unsigned blocks, unsigned thread, unsigned threads, F&& f) {
    const unsigned step = blocks * threads * U;
    for (unsigned base = block * threads * U; base < n; base += step) f(base + thread);
}

}  // namespace tss
