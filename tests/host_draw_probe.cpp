// Walks a draw list as the raster's warps do and prints how often each sample is
// drawn; tests/test_draw_split.py checks it. No GPU: the list's arithmetic only.
// Arguments: warps, then (items, samples per item) pairs.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <vector>

#include "rb_kernels.h"

int main(int argc, char** argv) {
    const uint32_t warps = (uint32_t)std::strtoul(argv[1], nullptr, 10);
    std::vector<rb::DrawItem> items;
    std::vector<uint32_t> count;
    unsigned long long total = 0;
    for (int a = 2; a + 1 < argc; a += 2)
        for (unsigned long k = std::strtoul(argv[a], nullptr, 10); k > 0; k--) {
            count.push_back((uint32_t)std::strtoul(argv[a + 1], nullptr, 10));
            items.push_back(rb::drawItem((uint32_t)(0x1FFFFFu - items.size()), total));
            total += count.back();
        }
    std::vector<unsigned long long> next(items.size(), 0);  // samples drawn of each item, in order
    unsigned long long drawn = 0, bad = 0;
    for (uint32_t w = 0; w < warps; w++) {
        const rb::DrawShare share = rb::drawShare(total, warps, w);
        if (share.begin >= share.end) continue;
        size_t lo = 0;
        for (size_t hi = items.size(); hi - lo > 1;) {
            const size_t mid = (lo + hi) / 2;
            (rb::itemFirst(items[mid]) <= share.begin ? lo : hi) = mid;
        }
        for (unsigned long long s = share.begin; s < share.end; lo++) {
            if (lo >= items.size() || rb::itemNode(items[lo]) != 0x1FFFFFu - lo) {
                bad++;
                break;
            }
            const uint32_t stop = rb::itemStop(items[lo], count[lo], share.end);
            const unsigned long long from = s - rb::itemFirst(items[lo]);
            if (from != next[lo] || stop > count[lo] || from > stop) bad++;
            next[lo] = stop;
            drawn += stop - from;
            s = rb::itemFirst(items[lo]) + stop;
        }
    }
    std::printf("%llu %llu %llu\n", total, drawn, bad);
    return 0;
}
