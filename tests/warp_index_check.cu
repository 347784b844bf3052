// Host-only check of warpOf (race_gb300/csrc/sweep_ops.cuh): for launches of
// 256 threads a block and a warp per row, prints the row counts at which a
// row would be run by another warp than its own. Built and run by
// tests/test_zz_index_range.py without a GPU; test infrastructure only.
#include <cstdio>
#include <cstdlib>

#include "sweep_ops.cuh"

int main(int argc, char **argv) {
    int bad = 0;
    for (int i = 1; i < argc; ++i) {
        const long long n = atoll(argv[i]);
        const int blocks = race::ceilDiv(32 * n, 256);
        bool ok = 8LL * blocks >= n;
        for (long long r : {0LL, n / 2, n - 1})
            for (unsigned lane : {0u, 31u})
                ok &= race::warpOf((unsigned)(r / 8), 256, (unsigned)(r % 8) * 32 + lane) == r;
        for (unsigned lane : {0u, 255u}) ok &= race::warpOf(blocks - 1, 256, lane) >= 8LL * (blocks - 1);
        if (!ok) printf("%lld\n", n);
        bad |= !ok;
    }
    return bad;
}
