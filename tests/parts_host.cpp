/* Every ray of the mixed trace's queue followed from part to lane (lensParts.h), over frames from one tile to
 * thousands, launch shapes, limits of rays a warp and numbers of heavy slots. */
#include "lensParts.h"

#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

using namespace artf;

static long checked = 0, wrong = 0;
static void check(bool ok) { ++checked, wrong += !ok; }

template <bool kSplit> static void follow(int units, const MixedGrid& g, unsigned heavySlots) {
    const MixedParts q = partsOf<kSplit>((unsigned)units, heavySlots, (unsigned)g.mostHeavy, g.lanesLog2);
    std::vector<int> seen((size_t)units, 0);
    std::vector<unsigned> started; /* a slot's first part, to see that the order's slots start in their order */
    for (unsigned part = 0; part < q.parts; ++part) {
        int rays = -1;
        const unsigned first = partFirst<kSplit>(q, part, g.lanesLog2, rays);
        check(rays >= 0 && rays <= 5 && (first & 31u) + (1u << rays) <= 32u); /* within one slot */
        if (!(first & 31u)) started.push_back(first >> 5);
        for (unsigned lane = 0; lane < 32u; ++lane)
            if (lane >> rays == 0) {
                check(first + lane < (unsigned)units);
                if (first + lane < (unsigned)units) ++seen[first + lane];
            }
    }
    check(std::all_of(seen.begin(), seen.end(), [](int n) { return n == 1; }));
    check(std::is_sorted(started.begin(), started.end()) && started.size() == (size_t)units / 32);
    check(q.heavy <= heavySlots * 32 && q.heavy <= (unsigned)g.mostHeavy * 32);
}

int main() {
    std::mt19937 rng(4);
    const int sms[] = {1, 3, 152}, blocks[] = {32, 64, 96, 128, 192, 256}, refills[] = {0, 1, 2, 3, 5, 8, 16, 31, 32};
    for (int sm : sms)
        for (int block : blocks)
            for (int refill : refills)
                for (int size = 0; size < 24; ++size) {
                    const int perSm = (int)(rng() % 5), warps = std::max(perSm, 1) * sm * (block / 32);
                    /* one slot, the sizes about one, three and six slots a warp, and any */
                    const int about[] = {1, warps, 3 * warps, 6 * warps, 7 * warps, 1 + (int)(rng() % 2000u)};
                    const int slots = std::min(2500, std::max(1, about[size % 6] + (int)(rng() % 5u) - 2)), units = slots * 32;
                    const MixedGrid g = mixedGridOf(units, block, perSm, sm, refill);
                    check(g.blocks >= 1 && g.blocks <= g.most && g.most * (block / 32) == warps);
                    check(g.lanesLog2 >= 0 && g.lanesLog2 <= 5 && (refill == 0 || 1 << g.lanesLog2 <= refill));
                    check(g.resident == (units >> g.lanesLog2 <= warps));
                    /* as many warps as parts, or every warp that fits */
                    check((long long)g.blocks * (block / 32) >= std::min<long long>(units >> g.lanesLog2, warps));
                    check(g.mostHeavy >= 0 && (g.mostHeavy == 0 || (g.lanesLog2 == 5 && slots < 6 * warps)));
                    follow<false>(units, g, 0);
                    if (g.mostHeavy > 0)
                        for (unsigned heavy : {0u, 1u, (unsigned)slots / 3, (unsigned)slots}) follow<true>(units, g, heavy);
                }
    printf("checked %ld\nwrong %ld\n", checked, wrong);
    return 0;
}
