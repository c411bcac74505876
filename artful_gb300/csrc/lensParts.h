/* artful_cuda — how the mixed trace's rays are shared among warps: the launch's grid, how many rays a warp takes at
 * a time, and which rays a part of the queue is.  Whole numbers alone, for the kernels, their launch and a host test
 * that follows every ray. */
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define ARTF_PART __host__ __device__ __forceinline__
#else
#define ARTF_PART inline
#endif

namespace artf {

constexpr int kHeavyRaysLog2 = 3; /* a heavy slot's parts: eight rays */

/* The persistent grid, and how many rays a warp takes at a time: all of a slot's 32 while that gives every
 * resident warp one; for a frame too small for that, half as many, and so on, down to two, so that more
 * warps share the rays and each has fewer that part ways (a warp runs what any of its rays needs, and
 * rays of a small frame's neighbouring pixels part early: a 101 x 67 frame took 119 us by 32 rays, 84 by
 * 8, 80 by 4 or 2; at 1920 x 1080 a warp's 32 rays stay together, 30.2 of 32 lanes busy).  refillBatch
 * sets the most.
 * Heavy slots are split where warps take whole slots of 32, the fewer the more slots there are: a quarter of
 * the warps' number at three slots a warp, none from six on (us, whole slots against split: 320 x 180 99 and
 * 79, 384 x 216 104 and 80, 512 x 288 126 and 101, 640 x 360 114 and 97, 320 x 180 x 4 rays 155 and 115, 768 x
 * 432 180 and 156; at 960 x 540, 6.7 slots a warp, 143 and 150; at 1280 x 720, 11.8, splitting 304 slots 181
 * and 188). */
struct MixedGrid {
    int blocks, most, lanesLog2; /* the launch's blocks, and as many as are resident at once */
    bool resident; /* every part has a warp at once: the order they start in makes no difference */
    int mostHeavy; /* the heavy slots that are split at most, for a trace that orders its slots */
};

inline MixedGrid mixedGridOf(int totalUnits, int block, int perSm, int smCount, int refillBatch) {
    const long long grid = (long long)(perSm > 0 ? perSm : 1) * smCount, warps = grid * (block / 32);
    MixedGrid g;
    g.lanesLog2 = 5;
    while (refillBatch > 0 && 1 << g.lanesLog2 > refillBatch) --g.lanesLog2;
    while (g.lanesLog2 > 1 && (long long)(totalUnits >> g.lanesLog2) * 2 <= warps) --g.lanesLog2;
    const long long parts = totalUnits >> g.lanesLog2, needed = (parts * 32 + block - 1) / block;
    const long long slots = totalUnits >> 5, room = (6 * warps - slots) / 12;
    g.mostHeavy = room > 0 && g.lanesLog2 == 5 ? (int)room : 0;
    g.resident = parts <= warps;
    g.most = (int)grid;
    g.blocks = (int)(grid > needed ? needed : grid);
    if (g.blocks < 1) g.blocks = 1;
    return g;
}

/* The queue's parts: the first `heavy` rays, those of the heavy slots, eight at a time (kSplit), the rest
 * 2^lanesLog2 at a time. */
struct MixedParts {
    unsigned heavy, heavyParts, parts;
};
template <bool kSplit> ARTF_PART MixedParts partsOf(unsigned totalUnits, unsigned heavySlots, unsigned mostHeavy, int lanesLog2) {
    MixedParts q;
    q.heavy = kSplit ? (heavySlots < mostHeavy ? heavySlots : mostHeavy) << 5 : 0u;
    q.heavyParts = q.heavy >> kHeavyRaysLog2;
    q.parts = q.heavyParts + ((totalUnits - q.heavy) >> lanesLog2);
    return q;
}
/* A part's first ray, and how many follow (their number's logarithm): within one slot. */
template <bool kSplit> ARTF_PART unsigned partFirst(const MixedParts& q, unsigned part, int lanesLog2, int& rays) {
    const bool split = kSplit && part < q.heavyParts;
    rays = split ? kHeavyRaysLog2 : lanesLog2;
    return split ? part << rays : q.heavy + ((part - q.heavyParts) << rays);
}

}  // namespace artf
