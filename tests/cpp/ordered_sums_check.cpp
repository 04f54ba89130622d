// The resident PCG's ordered sums (csrc/pcg_resident.cu, ORDERED) over every
// size and SM count a plan may meet: where ordered_sums_fit takes a layout, the
// kernel's warp tasks reach each component of each part's blocks once.  Prints
// "ok" or the first layout that loses or repeats one.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "internal.h"

using namespace mfem;

// Every component of the parts' blocks summed exactly once.
static bool covers(const ResidentHost &h, int n, int cluster, bool grid) {
    const int bw = ordered_block_warps(n, h.blocks), tasks = !grid && cluster > 1 ? kPartTasks : 1;
    for (const ResPart &P : h.parts) {
        auto row = [&](int b) { return (int)((long long)n * (P.block_lo + b) / h.blocks); };
        if (!grid && cluster <= 1 && P.nblocks > 2) return false;
        std::vector<int> met(3 * P.nown, 0);
        for (int w = 0; w < kPartWarps; ++w)
            for (int q = 0; q < tasks; ++q) {
                const int t = w + kPartWarps * q, b = t / bw, wi = t - b * bw;
                if (b >= P.nblocks) break;
                const int end = 3 * (row(b + 1) - row(0));
                for (int lane = 0; lane < 32; ++lane)
                    for (int i = 3 * (row(b) - row(0)) + 32 * wi + lane; i < end; i += kPartThreads) {
                        ++met[i];
                        if (!grid) break;  // one component a lane off the grid
                    }
            }
        for (int m : met)
            if (m != 1) return false;
    }
    return true;
}

int main() {
    std::vector<int32_t> rp(30001), ci(30000);
    for (int i = 0; i < 30000; ++i) rp[i] = ci[i] = i;
    rp[30000] = 30000;
    int taken = 0;
    for (int sms : {1, 2, 7, 16, 18, 36, 64, 97, 98, 99, 108, 132, 148, 152, 160})
        for (int n = 1; n <= 30000; n += n < 400 ? 1 : n < 6600 ? 13 : 997)
            for (int grid = 0; grid < 2; ++grid) {
                // as the plan chooses them
                const int blocks = std::max(1, std::min(sms, (n + 63) / 64));
                const int parts = grid ? blocks : std::min(kPartMaxCluster, (blocks + 1) / 2);
                if (!grid && n > 6400) continue;
                ResidentHost h;
                resident_add_ranges(h, rp.data(), ci.data(), n, parts, blocks, false);
                if (h.nown_max > kPartThreads) continue;
                const bool fit = ordered_sums_fit(h, parts, grid != 0);
                const bool all = covers(h, n, parts, grid != 0);
                if (fit && !all) {
                    printf("%d SMs, %d rows, %d parts, %d blocks%s: components lost\n", sms, n, parts, blocks,
                           grid ? " (grid)" : "");
                    return 1;
                }
                // nothing that works on a whole GPU is refused
                if (!fit && all && sms >= 132 && h.block_max <= (grid ? 1 : kPartMaxBlocks)) {
                    printf("%d SMs, %d rows, %d parts, %d blocks: refused\n", sms, n, parts, blocks);
                    return 1;
                }
                taken += fit;
            }
    if (taken < 1000) return 1;
    puts("ok");
    return 0;
}
