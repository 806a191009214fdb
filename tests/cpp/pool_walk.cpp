// Walks the shares of all warps of a point pool (pool_share.cuh) on the host,
// each in takes of its own sizes, and checks that every point of the batch is
// taken exactly once.  Arguments: blocks of 128 threads, points, seed.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "pool_share.cuh"

int main(int argc, char** argv) {
    if (argc != 4) return 2;
    const uint64_t blocks = strtoull(argv[1], nullptr, 10), n = strtoull(argv[2], nullptr, 10);
    uint32_t rnd = (uint32_t)strtoul(argv[3], nullptr, 10) * 2654435761u + 1u;
    std::vector<uint8_t> taken(n, 0);
    const uint64_t stride = 128 * blocks;
    for (uint64_t first = 0; first < stride && first < n; first += 32) {
        cg::PoolShare share(first, stride, n);
        // A third of the warps take whole groups, a third as lanes end, a third
        // change over after some points.
        const uint32_t kind = (first / 32) % 3;
        const uint32_t change = kind == 0 ? 0 : kind == 1 ? ~0u : share.end / 3;
        while (share.next < share.end) {
            rnd = rnd * 1664525u + 1013904223u;
            const uint32_t take = share.next < change && share.next ? 1 + (rnd >> 16) % 32 : 32;
            for (uint32_t j = 0; j < take; ++j) {
                const uint64_t i = share.index(j);
                if (i < n) ++taken[i];
            }
            share.advance(take);
        }
    }
    for (uint64_t i = 0; i < n; ++i)
        if (taken[i] != 1) {
            printf("point %llu taken %d times\n", (unsigned long long)i, taken[i]);
            return 1;
        }
    return 0;
}
