/* artful_cuda — a traced frame to what a screen shows: the bloom pyramid and the tone map with its
 * dither, on the GPU.  Restates the software backend's bloomDownRow / bloomUpRow / bloomTap
 * (src/software/software.c:320-387) and lensToneMap / lensFill (src/software/lens.inc:387-440), with
 * the same float operations in the same order: built with the exact flags (no contraction, IEEE
 * division and square root), the BGRA frame comes out bit for bit the software backend's.
 *
 * The pyramid's levels are the frame's bloom table (ArtfCudaHoleFrame.bloom: offset, width, height),
 * three float planes of the frame's bloom pixel count.  Level 0 takes the mean of four pixels' light
 * above the threshold (2) and under the ceiling (48); each next level four bilinear taps of the one
 * before; then each level, from the top down, adds four taps of the one above, times 0.85.  The tone
 * map reads level 0 between its texels, turns its glow toward grey (0.9), adds it times bloom * 0.15,
 * scales by the exposure, applies Narkowicz's ACES fit and a square root, and dithers by a hash. */
#include "nvtxRange.h"
#include "artful_cuda.h"

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

namespace {

constexpr float kThreshold = 2.f, kCeiling = 48.f, kFade = .85f, kWhite = .9f;

__device__ __forceinline__ float minRef(float a, float b) { return b < a ? b : a; } /* core.h artfMinf */
__device__ __forceinline__ float maxRef(float a, float b) { return a < b ? b : a; } /* core.h artfMaxf */
__device__ __forceinline__ int clampRef(int v, int lo, int hi) { return v < lo ? lo : v > hi ? hi : v; }
__device__ __forceinline__ float minX(float a, float b) { return a < b ? a : b; }   /* simd.h v8fMin */

__device__ __forceinline__ float bright(float v) { return minRef(maxRef(v - kThreshold, 0.f), kCeiling); }

struct Planes {
    float* c[3];
};

/* The pass is a chain of short kernels, so each may start while the one before it drains (programmatic
 * dependent launch) and waits here, before its first read, until that one has finished and its writes are
 * visible.  Since a kernel of the chain finishes only after the one before it, so has all before them. */
__device__ __forceinline__ void chained() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... P, typename... A>
cudaError_t follow(cudaStream_t stream, void (*kernel)(P...), dim3 grid, int block, const A&... args) {
    cudaLaunchAttribute early;
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid, c.blockDim = dim3((unsigned)block), c.stream = stream, c.attrs = &early, c.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, kernel, P(args)...);
    if (e != cudaSuccess) (void)cudaGetLastError(); /* (or the next launch's check would report it) */
    return e;
}

/* software.c:334-351: level 0 from the frame's light. */
__global__ void bloomFirst(const float4* hdr, int width, int height, Planes bloom, uint32_t at, int toW, int toH) {
    chained();
    const int x = (int)(blockIdx.x * blockDim.x + threadIdx.x), y = (int)blockIdx.y;
    if (x >= toW || y >= toH) return;
    const int lastX = width - 1, lastY = height - 1;
    const int y0 = min(y * 2, lastY), y1 = min(y * 2 + 1, lastY), x0 = min(x * 2, lastX), x1 = min(x * 2 + 1, lastX);
    const float4 a0 = hdr[(size_t)y0 * width + x0], a1 = hdr[(size_t)y0 * width + x1];
    const float4 b0 = hdr[(size_t)y1 * width + x0], b1 = hdr[(size_t)y1 * width + x1];
    const float s[3][4] = {{a0.x, a1.x, b0.x, b1.x}, {a0.y, a1.y, b0.y, b1.y}, {a0.z, a1.z, b0.z, b1.z}};
    for (int c = 0; c < 3; ++c)
        bloom.c[c][at + (size_t)y * toW + x] = (bright(s[c][0]) + bright(s[c][1]) + bright(s[c][2]) + bright(s[c][3])) * .25f;
}

/* software.c:320-328 bloomTap reads a level bilinearly at a place in its texels, clamped at the edges: between
 * a and b, a part of the way. */
__device__ __forceinline__ float between(float a, float b, float part) { return a + (b - a) * part; }

/* software.c:353-365: a texel of level L from level L - 1, four taps at 2 x + .5 +- 1 and 2 y + .5 +- 1: each
 * halfway between two columns and two rows, so the four by four texels from (2 x - 1, 2 y - 1) on. */
__device__ __forceinline__ float downTexel(const float* from, int fromW, int fromH, int x, int y) {
    int column[4];
    float row[4][2];
#pragma unroll
    for (int k = 0; k < 4; ++k) column[k] = clampRef(2 * x - 1 + k, 0, fromW - 1);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float* at = from + (size_t)clampRef(2 * y - 1 + k, 0, fromH - 1) * fromW;
        row[k][0] = between(at[column[0]], at[column[1]], .5f), row[k][1] = between(at[column[2]], at[column[3]], .5f);
    }
    float sum = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) sum += between(row[k & 2][k & 1], row[(k & 2) + 1][k & 1], .5f);
    return sum * .25f;
}

/* software.c:368-386: what the texels (2 m, 2 n) .. (2 m + 1, 2 n + 1) of level L gain, four taps of level L + 1
 * each, at x / 2 - .25 +- .5 and so in y: a quarter of the way between two texels for an even x, three quarters
 * for an odd one, the same three columns and rows around (m, n) for all four: 9 texels read where 16 taps read
 * 64 (1080p: the largest level's launch 11.4 -> 9.2 us, most of the rest its launch; with the levels down and
 * the tone map's pairs of pixels, 20 -> 18 us and bound by its instructions, the frame 523 -> 513). */
__device__ __forceinline__ void upTexels(const float* from, int fromW, int fromH, int m, int n, float gain[2][2]) {
    float a[3][3];
    int column[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) column[k] = clampRef(m - 1 + k, 0, fromW - 1);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const float* at = from + (size_t)clampRef(n - 1 + j, 0, fromH - 1) * fromW;
#pragma unroll
        for (int k = 0; k < 3; ++k) a[j][k] = at[column[k]];
    }
#pragma unroll
    for (int odd = 0; odd < 2; ++odd) {
        float row[3][2];
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k) row[j][k] = between(a[j][k], a[j][k + 1], odd ? .75f : .25f);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float sum = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) sum += between(row[k >> 1][k & 1], row[(k >> 1) + 1][k & 1], i ? .75f : .25f);
            gain[i][odd] = sum * (.25f * kFade);
        }
    }
}

__device__ __forceinline__ void addTexels(float* level, int width, int height, int m, int n, const float gain[2][2]) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (2 * m + k < width && 2 * n + i < height) level[(size_t)(2 * n + i) * width + 2 * m + k] += gain[i][k];
}

/* A thread a texel of one plane (blockIdx.z). */
__global__ void bloomDown(const __grid_constant__ Planes bloom, uint32_t fromAt, int fromW, int fromH, uint32_t toAt, int toW, int toH) {
    chained();
    const int x = (int)(blockIdx.x * blockDim.x + threadIdx.x), y = (int)blockIdx.y;
    if (x >= toW || y >= toH) return;
    float* const plane = bloom.c[blockIdx.z];
    plane[toAt + (size_t)y * toW + x] = downTexel(plane + fromAt, fromW, fromH, x, y);
}

/* A thread four texels of one plane. */
__global__ void bloomUp(const __grid_constant__ Planes bloom, uint32_t fromAt, int fromW, int fromH, uint32_t toAt, int toW, int toH) {
    chained();
    const int m = (int)(blockIdx.x * blockDim.x + threadIdx.x), n = (int)blockIdx.y;
    if (2 * m >= toW || 2 * n >= toH) return;
    float* const plane = bloom.c[blockIdx.z];
    float gain[2][2];
    upTexels(plane + fromAt, fromW, fromH, m, n, gain);
    addTexels(plane + toAt, toW, toH, m, n, gain);
}

/* The pyramid's small levels, `first` to the last, down and up again in one block's shared memory: a launch
 * each is some 3 us, most of it waiting for the one before.  Up to 1024 texels in all (a 1080p frame's last
 * three levels, 8 us: the frame 535 -> 525 us; 256 to 2048 are alike); 4096 keep the one block longer than their
 * launches take (517 against 513). */
constexpr int kTailThreads = 1024;
constexpr size_t kTailTexels = 1024;
struct TailLevels {
    uint32_t level[ARTF_CUDA_BLOOM_LEVELS][4];
    int first, count;
};

__global__ void __launch_bounds__(kTailThreads) bloomTail(const __grid_constant__ Planes bloom, const __grid_constant__ TailLevels t) {
    __shared__ float held[3 * kTailTexels];
    chained();
    const uint32_t base = t.level[t.first][0], texels = t.level[t.count - 1][0] - base +
                                                        t.level[t.count - 1][1] * t.level[t.count - 1][2];
    for (int i = t.first; i < t.count; ++i) {
        const int w = (int)t.level[i][1], h = (int)t.level[i][2], fw = (int)t.level[i - 1][1], fh = (int)t.level[i - 1][2];
        for (int k = (int)threadIdx.x; k < 3 * w * h; k += kTailThreads) {
            const int c = k / (w * h), at = k - c * w * h, y = at / w, x = at - y * w;
            const float* from = i == t.first ? bloom.c[c] + t.level[i - 1][0]
                                             : held + c * texels + (t.level[i - 1][0] - base);
            held[c * texels + (t.level[i][0] - base) + at] = downTexel(from, fw, fh, x, y);
        }
        __syncthreads();
    }
    for (int i = t.count - 1; i-- > t.first;) {
        const int w = (int)t.level[i][1], h = (int)t.level[i][2], fw = (int)t.level[i + 1][1], fh = (int)t.level[i + 1][2];
        const int ms = (w + 1) / 2, ns = (h + 1) / 2;
        for (int k = (int)threadIdx.x; k < 3 * ms * ns; k += kTailThreads) {
            const int c = k / (ms * ns), at = k - c * ms * ns, n = at / ms, m = at - n * ms;
            float gain[2][2];
            upTexels(held + c * texels + (t.level[i + 1][0] - base), fw, fh, m, n, gain);
            addTexels(held + c * texels + (t.level[i][0] - base), w, h, m, n, gain);
        }
        __syncthreads();
    }
    for (uint32_t k = threadIdx.x; k < 3 * texels; k += kTailThreads) bloom.c[k / texels][base + k % texels] = held[k];
}

/* lens.inc:56-61: the dither's hash (the star lattice's). */
__device__ __forceinline__ uint32_t hash3(uint32_t x, uint32_t y, uint32_t z) {
    uint32_t h = x * 73856093u ^ y * 19349663u ^ z * 83492791u;
    h = (h ^ h >> 15) * 0x2C1B3C6Du;
    h = (h ^ h >> 12) * 0x297A2D39u;
    return h ^ h >> 15;
}

/* lens.inc:387-391: Narkowicz's fit to ACES, and a square root for the screen. */
__device__ __forceinline__ float toneCurve(float x) {
    const float top = x * (x * 2.51f + .03f);
    const float bottom = x * (x * 2.43f + .59f) + .14f;
    return sqrtf(minX(top / bottom, 1.f));
}

/* lens.inc:395-440: light plus glow, exposed, tone mapped and dithered to premultiplied BGRA.  A thread two
 * pixels side by side, 2 m and 2 m + 1: their glow lies three quarters of the way from texel m - 1 to m and a
 * quarter from m to m + 1. */
__global__ void toneMap(const float4* hdr, int width, int height, Planes bloom, uint32_t at, int bw, int bh,
                        float exposure, float spread, uint32_t* bgra) {
    chained();
    const int m = (int)(blockIdx.x * blockDim.x + threadIdx.x), y = (int)blockIdx.y;
    if (2 * m >= width || y >= height) return;
    const int n = y >> 1;
    const float partY = y & 1 ? .25f : .75f;
    const int y0 = clampRef(y & 1 ? n : n - 1, 0, bh - 1), y1 = clampRef(y & 1 ? n + 1 : n, 0, bh - 1);
    int column[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) column[k] = clampRef(m - 1 + k, 0, bw - 1);
    const float4* const lit = hdr + (size_t)y * width + 2 * m;
    const float4 light4[2] = {lit[0], 2 * m + 1 < width ? lit[1] : make_float4(0.f, 0.f, 0.f, 0.f)};
    float glows[2][3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float *r0 = bloom.c[c] + at + y0 * bw, *r1 = bloom.c[c] + at + y1 * bw;
        const float a[3] = {r0[column[0]], r0[column[1]], r0[column[2]]}, d[3] = {r1[column[0]], r1[column[1]], r1[column[2]]};
#pragma unroll
        for (int k = 0; k < 2; ++k)
            glows[k][c] = between(between(a[k], a[k + 1], k ? .25f : .75f), between(d[k], d[k + 1], k ? .25f : .75f), partY);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int x = 2 * m + k;
        if (x >= width) return;
        const float grey = glows[k][0] * .3f + glows[k][1] * .59f + glows[k][2] * .11f;
        const float light[3] = {light4[k].x, light4[k].y, light4[k].z};
        const float dither = (float)(int)(hash3((uint32_t)(x + y * 8192), 7u, 13u) & 255u) * (1.f / 255.f);
        uint32_t bytes[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float glow = glows[k][c] + (grey - glows[k][c]) * kWhite;
            const float shown = toneCurve((light[c] + glow * spread) * exposure);
            bytes[c] = (uint32_t)(int)minX(shown * 255.f + dither, 255.f);
        }
        bgra[(size_t)y * width + x] = bytes[0] << 16 | bytes[1] << 8 | bytes[2] | 0xFF000000u;
    }
}

}  // namespace

/* The pyramid and tone map of one frame; bloom: three planes of the frame's bloom pixel count. */
extern "C" int artfCudaPostLaunch(const ArtfCudaHoleFrame* frame, const float* hdr, float* const bloomPlanes[3],
                                  uint32_t* bgra, void* stream) {
    artf::Range range("artfCudaPostLaunch");
    if (!frame || !hdr || !bloomPlanes || !bgra) return ARTF_CUDA_EINVAL;
    const int width = (int)frame->size[0], height = (int)frame->size[1], levels = (int)frame->size[3];
    if (width < 1 || height < 1 || levels < 1 || levels > ARTF_CUDA_BLOOM_LEVELS) return ARTF_CUDA_EINVAL;
    cudaStream_t s = (cudaStream_t)stream;
    Planes planes = {{bloomPlanes[0], bloomPlanes[1], bloomPlanes[2]}};
    const int block = 128;
    const uint32_t(*table)[4] = frame->bloom;
    cudaError_t e = cudaSuccess;
    /* the levels from `tail` on in one launch: from the second at the earliest, where they lie one after another
     * and fit the block, and there are two or more */
    int tail = levels;
    size_t texels = 0;
    for (int i = levels - 1; i > 0; --i) {
        texels += (size_t)table[i][1] * table[i][2];
        if (texels > kTailTexels || (i + 1 < levels && table[i][0] + table[i][1] * table[i][2] != table[i + 1][0])) break;
        tail = i;
    }
    if (levels - tail < 2) tail = levels;
    for (int i = 0; i < tail && e == cudaSuccess; ++i) {
        const dim3 grid((table[i][1] + block - 1) / block, table[i][2], i ? 3 : 1);
        if (i == 0) e = follow(s, bloomFirst, grid, block, (const float4*)hdr, width, height, planes, table[0][0],
                               (int)table[0][1], (int)table[0][2]);
        else e = follow(s, bloomDown, grid, block, planes, table[i - 1][0], (int)table[i - 1][1], (int)table[i - 1][2],
                        table[i][0], (int)table[i][1], (int)table[i][2]);
    }
    if (tail < levels && e == cudaSuccess) {
        TailLevels t;
        memcpy(t.level, table, sizeof t.level);
        t.first = tail, t.count = levels;
        e = follow(s, bloomTail, dim3(1), kTailThreads, planes, t);
    }
    for (int i = tail < levels ? tail : levels - 1; i-- > 0 && e == cudaSuccess;) {
        const dim3 grid(((table[i][1] + 1) / 2 + block - 1) / block, (table[i][2] + 1) / 2, 3);
        e = follow(s, bloomUp, grid, block, planes, table[i + 1][0], (int)table[i + 1][1], (int)table[i + 1][2],
                   table[i][0], (int)table[i][1], (int)table[i][2]);
    }
    const float spread = frame->look[3] * (1.f - kFade);
    if (e == cudaSuccess)
        e = follow(s, toneMap, dim3(((width + 1) / 2 + block - 1) / block, height), block, (const float4*)hdr, width, height, planes,
                   table[0][0], (int)table[0][1], (int)table[0][2], frame->image[0], spread, bgra);
    return e == cudaSuccess ? ARTF_CUDA_OK : ARTF_CUDA_ELAUNCH;
}
