/* artful_cuda — the trace kernels, generic in the arithmetic type.  Included by lensExact.cu,
 * lensFast.cu and lensFp64.cu, whose compile flags fix how float rounds.
 *
 * Work layout: a warp owns an 8 x 4 tile of pixels (rays of neighbouring pixels bend alike, so the
 * lanes of a warp take similar numbers of steps and cross the disc at similar moments), a thread owns
 * one pixel and traces its rays one after the other, summing them in the reference's order.  The HDR
 * frame is width * height float4: linear RGB and the pixel's class bits.  A persistent variant, where
 * each warp pulls tiles from a device queue, lives in the same file. */
#pragma once

#include "lensCore.cuh"
#include "lensLaunch.h"

namespace artf {
namespace {

template <typename R> struct KernelParams {
    Frame<R> f;                 /* the frame in R: kernel parameters sit in the constant bank */
    ArtfCudaHoleFrame h;        /* sample positions come from the FP32 frame, as the reference's */
    const float* map;
    const float* fluid;
    float4* hdr;
    ArtfCudaRayEnd* ends;
    unsigned long long* counters;
    int jitter;
    uint32_t seed;
    R stepScale;
    int maxSteps;
    int rays;
    float share;
    int tilesX, tiles;          /* 8 x 4 pixel tiles: this launch's count */
    int tileBegin;              /* the first (a band of the frame starts further down) */
    int lanesLog2;              /* a warp takes 2^lanesLog2 of a tile's pixels: a part of it */
};

/* What a thread counts, reduced over the warp before it reaches the device counters. */
struct Tally {
    unsigned rays = 0, steps = 0, crossings = 0, escapes = 0;
};

__device__ __forceinline__ void flushTally(const Tally& t, unsigned long long* counters) {
    const unsigned rays = __reduce_add_sync(0xFFFFFFFFu, t.rays);
    const unsigned steps = __reduce_add_sync(0xFFFFFFFFu, t.steps);
    const unsigned crossings = __reduce_add_sync(0xFFFFFFFFu, t.crossings);
    const unsigned escapes = __reduce_add_sync(0xFFFFFFFFu, t.escapes);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(counters + CRays, (unsigned long long)rays);
        atomicAdd(counters + CSteps, (unsigned long long)steps);
        atomicAdd(counters + CCrossings, (unsigned long long)crossings);
        atomicAdd(counters + CEscapes, (unsigned long long)escapes);
    }
}

__device__ __forceinline__ unsigned classBits(unsigned kind) {
    unsigned bits = (kind & ARTF_CUDA_END_LIT) ? 1u : 0u;
    if ((kind & 15u) == ARTF_CUDA_END_SKY) bits |= 2u;
    else if (!(kind & ARTF_CUDA_END_LIT)) bits |= 4u;
    return bits;
}

/* What a thread counts over its rays, in shared memory: touched once a ray, it would hold registers
 * through the stepping loop. */
enum { kTallyRays, kTallySteps, kTallyCrossings, kTallyEscapes, kTallyCount };
typedef unsigned Tallies[kTallyCount][256];

__device__ __forceinline__ void clearTallies(Tallies& t) {
    for (int k = 0; k < kTallyCount; ++k) t[k][threadIdx.x] = 0;
}
/* A warp's tallies to the launch's counters; the whole warp calls it. */
__device__ __forceinline__ void flushTallies(const Tallies& t, unsigned long long* counters) {
    __syncwarp();
    const int to[kTallyCount] = {CRays, CSteps, CCrossings, CEscapes};
    for (int k = 0; k < kTallyCount; ++k) {
        const unsigned n = __reduce_add_sync(0xFFFFFFFFu, t[k][threadIdx.x]);
        if ((threadIdx.x & 31) == 0 && n) atomicAdd(counters + to[k], (unsigned long long)n);
    }
}

/* A finished ray's tallies and the rest of its end record. */
__device__ __forceinline__ void finishRay(int steps, unsigned crossings, unsigned kind, int wide, ArtfCudaRayEnd* end,
                                          Tallies& t) {
    const unsigned add[kTallyCount] = {1u, (unsigned)steps, crossings, (kind & 15u) == ARTF_CUDA_END_SKY ? 1u : 0u};
    for (int k = 0; k < kTallyCount; ++k) t[k][threadIdx.x] += add[k];
    if (end) {
        end->steps = (uint16_t)steps;
        end->crossings = (uint8_t)(crossings > 255u ? 255u : crossings);
        end->kind = (uint8_t)kind;
        end->fp64Steps = (uint16_t)wide;
        end->reserved = 0;
    }
}

/* One ray, from its image position to its end (lens.inc:99-351).  Adds its light to sum (3). */
template <typename R>
__device__ __forceinline__ unsigned traceRay(const KernelParams<R>& p, R nx, R ny, R time, R* sum,
                                             ArtfCudaRayEnd* end, Tallies& t) {
    const Frame<R>& f = p.f;
    RayConst<R> c;
    RayState<R> s;
    rayStart(f, nx, ny, time, p.stepScale, c, s);
    const R a = f.a, a2 = a * a;
    if (a != R(0)) s.drag = dragAt(a, a2, c.xiA, s.u);
    const R rhoScale = recipR(R(1) - divR(f.inner, f.outer));

    R raySum[3] = {R(0), R(0), R(0)}, through = R(1);
    unsigned kind = ARTF_CUDA_END_CAP, crossings = 0;
    if (end) {
        end->hitR = end->hitPhi = NAN;
        for (int k = 0; k < 3; ++k) end->dir[k] = 0.f;
        end->mino = (float)(R(p.maxSteps) * c.step);
    }
    int i = 0;
    while (i < p.maxSteps) {
        StepOut<R> o;
        nystromStep(a, c, s, o);
        ++i;
        /* (most steps meet nothing, which one branch decides) */
        if ((s.n[2] * o.next.n[2] < R(0)) | (R(0) > o.next.u) | (o.next.u > f.uHorizon)) {
            Crossing<R> x;
            bool opaque = false;
            if (crossingOf(f, rhoScale, c, s, o, x)) {
                ++crossings;
                R turn;
                const R light = shadeCrossing(f, rhoScale, p.map, p.fluid, c, x, through, raySum, &turn);
                if (light > R(0) && !(kind & ARTF_CUDA_END_LIT)) {
                    kind |= ARTF_CUDA_END_LIT;
                    if (end) end->hitR = (float)recipR(x.uc), end->hitPhi = (float)(turn - floorR(turn));
                }
                opaque = !(through > KF(.004)); /* (the transmission only changes here) */
            }
            if (R(0) > o.next.u) {
                const R part = divR(s.u, s.u - o.next.u);
                R away[3], dir[3];
                for (int k = 0; k < 3; ++k) away[k] = s.n[k] + part * (o.next.n[k] - s.n[k]);
                const R awayPsi = s.psi + part * (o.next.psi - s.psi);
                skyDirection(away, awayPsi, dir);
                if (f.stars > R(0)) shadeSky(f, p.map, c, dir, through, raySum);
                kind ^= ARTF_CUDA_END_CAP ^ ARTF_CUDA_END_SKY;
                if (end) {
                    for (int k = 0; k < 3; ++k) end->dir[k] = (float)dir[k];
                    end->mino = (float)((R(i - 1) + part) * c.step);
                }
                break;
            }
            const bool fell = o.next.u > f.uHorizon;
            if (fell || opaque) {
                kind ^= ARTF_CUDA_END_CAP ^ (fell ? ARTF_CUDA_END_HORIZON : ARTF_CUDA_END_OPAQUE);
                if (end) end->mino = (float)(R(i) * c.step);
                break;
            }
        }
        s = o.next;
    }
    for (int k = 0; k < 3; ++k) sum[k] = sum[k] + raySum[k];
    finishRay(i, crossings, kind, sizeof(R) == 8 ? i : 0, end, t);
    return kind;
}

/* All rays of one pixel, summed in the reference's order and scaled by 1 / rays (lens.inc:364-380). */
template <typename R> __device__ __forceinline__ void tracePixel(const KernelParams<R>& p, int32_t x, int32_t y,
                                                                  Tallies& t) {
    const size_t pixel = (size_t)y * (size_t)p.f.width + (size_t)x;
    R sum[3] = {R(0), R(0), R(0)};
    unsigned bits = 0;
    for (int k = 0; k < p.rays; ++k) {
        float nx, ny, moment;
        samplePosition(p.h, p.jitter, p.seed, x, y, k, &nx, &ny, &moment);
        const float time = p.h.disc[2] + p.h.spin[3] * moment;
        const int64_t endAt = (int64_t)pixel * p.rays + k;
        ArtfCudaRayEnd* end = p.ends && inBounds(p.f.fault, kBoundsRayEnd, endAt,
                                                 (int64_t)p.f.width * p.f.height * p.rays)
                                  ? p.ends + endAt
                                  : nullptr;
        bits |= classBits(traceRay(p, R(nx), R(ny), R(time), sum, end, t));
    }
    const R share = R(p.share);
    if (inBounds(p.f.fault, kBoundsPixel, (int64_t)pixel, (int64_t)p.f.width * p.f.height))
        p.hdr[pixel] = make_float4((float)(sum[0] * share), (float)(sum[1] * share), (float)(sum[2] * share), (float)bits);
}

/* A warp's part of this launch's tiles: pixels row by row, a thread each, 8 x 4 of them or fewer. */
template <typename R> __device__ __forceinline__ void tracePart(const KernelParams<R>& p, unsigned part, Tallies& t) {
    const int lane = threadIdx.x & 31;
    const unsigned first = part << p.lanesLog2, within = (first & 31u) + (unsigned)lane;
    const int tile = p.tileBegin + (int)(first >> 5);
    const int32_t x = (tile % p.tilesX) * 8 + (int32_t)(within & 7u), y = (tile / p.tilesX) * 4 + (int32_t)(within >> 3);
    if (lane >> p.lanesLog2 == 0 && x < p.f.width && y < p.f.height) tracePixel(p, x, y, t);
}

/* Blocks of 256 a SM the registers are cut for: 128 registers a thread in float (what the compiler takes by
 * itself, 80 in the exact trace, leaves a ray's stages too little in flight: 58.7 against 54.0 us for the
 * exact 320 x 180 frame, 1267 against 1225 for 1080p x 4; 168 and 96 are slower too); in double none (186:
 * 2381 against 2803 us at 128, 960 x 540). */
template <typename R> constexpr int kBlocks = sizeof(R) == 4 ? 2 : 1;

/* One warp per part, one thread per pixel. */
template <typename R> __global__ void __launch_bounds__(256, kBlocks<R>) traceTiles(const KernelParams<R> p) {
    const unsigned part = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    __shared__ Tallies t;
    clearTallies(t);
    if (part < (unsigned)p.tiles << 5 >> p.lanesLog2) tracePart(p, part, t);
    flushTallies(t, p.counters);
}

/* Persistent: a grid of resident warps that pull parts from the queue counter until none is left. */
template <typename R> __global__ void __launch_bounds__(256, kBlocks<R>) traceQueue(const KernelParams<R> p) {
    const unsigned parts = (unsigned)p.tiles << 5 >> p.lanesLog2;
    __shared__ Tallies t;
    clearTallies(t);
    for (;;) {
        unsigned part = 0;
        if ((threadIdx.x & 31) == 0) part = (unsigned)atomicAdd(p.counters + CQueue, 1ull);
        part = __shfl_sync(0xFFFFFFFFu, part, 0);
        if (part >= parts) break;
        tracePart(p, part, t);
        __syncwarp();
    }
    flushTallies(t, p.counters);
}

/* A list of rays at given image positions, one a thread (the per-ray entry point). */
struct RayList {
    int n;
    const float* nx;
    const float* ny;
    const float* time;
    float* rgb;
};

template <typename R> __global__ void __launch_bounds__(128) traceList(const KernelParams<R> p, const RayList l) {
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    __shared__ Tallies t;
    clearTallies(t);
    if (i < l.n) {
        R sum[3] = {R(0), R(0), R(0)};
        traceRay(p, R(l.nx[i]), R(l.ny[i]), R(l.time[i]), sum, p.ends ? p.ends + i : nullptr, t);
        for (int k = 0; k < 3; ++k) l.rgb[3 * i + k] = (float)sum[k];
    }
    flushTallies(t, p.counters);
}

template <typename R> cudaError_t launchUniform(const TraceLaunch& l, const void* frameSource) {
    KernelParams<R> p;
    if (sizeof(R) == 8) p.f.load(*(const ArtfCudaHoleFrame64*)frameSource, l.frame);
    else p.f.load(*(const ArtfCudaHoleFrame*)frameSource, l.frame);
    p.f.fault = l.counters + CBoundsKind;
    p.h = l.frame;
    p.map = l.map;
    p.fluid = l.fluid;
    p.hdr = l.hdr;
    p.ends = l.ends;
    p.counters = l.counters;
    p.jitter = l.jitter;
    p.seed = l.seed;
    p.stepScale = R(l.stepScale);
    p.maxSteps = l.stepScale < .75f ? 384 : 192;
    p.rays = l.jitter ? l.jitter : (int)(l.frame.size[2] * l.frame.size[2]);
    p.share = l.jitter ? 1.f / (float)l.jitter : l.frame.image[3];
    p.tilesX = ((int)l.frame.size[0] + 7) / 8;
    const int tileRows = ((int)l.frame.size[1] + 3) / 4;
    const int bandBegin = l.tileRows > 0 ? l.tileRowBegin : 0;
    const int bandRows = l.tileRows > 0 ? l.tileRows : tileRows;
    p.tileBegin = bandBegin * p.tilesX;
    p.tiles = p.tilesX * bandRows;
    p.lanesLog2 = 5;
    const int block = l.blockSize > 0 ? l.blockSize : 128;
    if (l.rayCount > 0) {
        const RayList list = {l.rayCount, l.rayX, l.rayY, l.rayTime, l.rayRgb};
        traceList<R><<<(l.rayCount + block - 1) / block, block, 0, l.stream>>>(p, list);
    } else {
        const void* kernel = l.persistent ? (const void*)traceQueue<R> : (const void*)traceTiles<R>;
        int perSm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, block, 0);
        const long long slots = (long long)(perSm > 0 ? perSm : 1) * l.smCount, warps = slots * (block / 32);
        /* A frame whose tiles leave half the GPU's warps without one is bound by its longest rays' latency:
         * its warps take half a tile each, and so on down to two pixels, and have fewer rays that part ways
         * (exact, 61 x 40: 76 -> 44 us; 200 x 112: 61 -> 54; FP32 160 x 90 x 4: 116 -> 89; parts for more
         * warps than there are cost more: 200 x 112 66 us).  In double a warp holds the FP64 pipe as long for
         * two lanes as for 32, so there parts are made up to eight warps a SM (61 x 40: 497 -> 325 us, 160 x
         * 90 547 -> 489). */
        const long long most = sizeof(R) == 4 ? warps : 8ll * l.smCount;
        while (p.lanesLog2 > 1 && ((long long)p.tiles << 5 >> p.lanesLog2) * 2 <= most) --p.lanesLog2;
        const long long blocks = (((long long)p.tiles << 5 >> p.lanesLog2) * 32 + block - 1) / block;
        if (l.persistent) traceQueue<R><<<(unsigned)(blocks < slots ? blocks : slots), block, 0, l.stream>>>(p);
        else traceTiles<R><<<(unsigned)blocks, block, 0, l.stream>>>(p);
    }
    return cudaGetLastError();
}

}  // namespace
}  // namespace artf
