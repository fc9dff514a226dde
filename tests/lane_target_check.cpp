/* lane_target against 64-bit arithmetic: the first, the last and random
 * threads of grids over up to 2^31 - 1 targets. */
#include <cstdint>
#include <cstdio>
#include <random>

#include "lq_lanes.h"

int main()
{
    std::mt19937_64 rng(5);
    const int64_t most = ((int64_t)1 << 31) - 1;
    for (unsigned lanes : {1u, 4u, 8u, 32u})
        for (int64_t n : {(int64_t)1, (int64_t)17, (int64_t)1 << 27, ((int64_t)1 << 29) - 1, ((int64_t)1 << 29) + 5,
                          most}) {
            const unsigned threads = 128;
            const int64_t blocks = (n * lanes + threads - 1) / threads;
            for (int k = 0; k < 2000; ++k) {
                const int64_t block = k == 0 ? 0 : k == 1 ? blocks - 1 : (int64_t)(rng() % (uint64_t)blocks);
                const unsigned thread = (unsigned)(rng() % threads);
                const int64_t want = (block * threads + thread) / lanes;
                if (want > most) continue;
                const int got = lqb::lane_target((unsigned)block, thread, threads, lanes);
                if (got != want) {
                    printf("lanes %u, %lld targets: block %lld thread %u gives %d, not %lld\n", lanes, (long long)n,
                           (long long)block, thread, got, (long long)want);
                    return 1;
                }
            }
        }
    printf("OK\n");
    return 0;
}
