// check_batch_kernel.cpp -- which kernel a batch launch takes, and with how many
// blocks (recurrence_blocks in mrg8g_tiles.h).
#include <cstdio>

#include "mrg8g_tiles.h"

using mrg8g::recurrence_blocks;

int main() {
    int bad = 0;
    const int sms = 152, occupancy = 9;
    for (int threads : {128, 256}) {
        const uint64_t wpb = threads / 32, resident = (uint64_t)sms * occupancy * wpb;
        for (uint64_t ntiles : {1ull, 4ull, 5ull, 1000ull, 1976ull, 1977ull, 5472ull, 5473ull, 100000ull, 4294967295ull})
            for (uint64_t longest : {1ull, 512ull, 513ull, 1024ull, 1025ull, 32768ull})
                for (bool one_kind : {false, true}) {
                    const bool small = (longest <= 512 && ntiles <= resident) ||
                                       (longest <= 1024 && one_kind && ntiles <= 13 * (uint64_t)sms);
                    const int free = recurrence_blocks(ntiles, longest, one_kind, threads, 0, occupancy, sms);
                    bad += (free > 0) != small;
                    // One warp per tile.
                    if (free) bad += (uint64_t)free * wpb < ntiles || ((uint64_t)free - 1) * wpb >= ntiles;
                    // A cap always runs the recurrence kernel, within it.
                    for (int cap : {1, 2, 4, 9, 1000}) {
                        const int b = recurrence_blocks(ntiles, longest, one_kind, threads, cap, occupancy, sms);
                        bad += b < 1 || b > sms * (cap < occupancy ? cap : occupancy);
                        bad += ((uint64_t)b - 1) * wpb >= ntiles;
                    }
                }
    }
    std::printf("bad=%d\n", bad);
    return bad != 0;
}
