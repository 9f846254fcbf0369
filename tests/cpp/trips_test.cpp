// Host check of the list kernels' index arithmetic (trips.hpp) with the launch shapes of
// the grid build, 2,432 blocks of 256 threads: the first and last blocks' trips over lists
// up to 2^31 - 1 entries take exactly the entries that are theirs, in order, and end.
// Prints "ok".
#include <cstdint>
#include <cstdio>
#include <initializer_list>

#include "../../twoscalesplit_gb300/csrc/trips.hpp"

template <int U>
bool check(unsigned n, unsigned block, unsigned blocks, unsigned thread, unsigned threads) {
    const uint64_t step = static_cast<uint64_t>(blocks) * threads * U;
    uint64_t want = static_cast<uint64_t>(block) * threads * U, trips = 0;
    bool ok = true;
    tss::for_trips<U>(n, block, blocks, thread, threads, [&](unsigned base) {
        ok = ok && want < n && base == want + thread;
        want += step;
        if (++trips > 4000000) std::printf("does not end\n"), throw 1;
    });
    return ok && want >= n;
}

int main() {
    const unsigned ns[] = {0u, 1u, 255u, 257u, 1024u, 622592u, 622593u, 2490369u, 2144993280u, 2144993281u,
                           2146000000u, 2146861057u, 2147483647u};
    for (unsigned n : ns)
        for (unsigned block : {0u, 1u, 1216u, 2430u, 2431u})
            for (unsigned thread : {0u, 31u, 255u})
                if (!check<1>(n, block, 2432, thread, 256) || !check<4>(n, block, 2432, thread, 256)) {
                    std::printf("n %u block %u thread %u\n", n, block, thread);
                    return 1;
                }
    std::printf("ok\n");
    return 0;
}
