/* artful_cuda — the reference's painted disc map, made on the GPU (src/scene/hole.c:14-197 buildDisc and
 * setRings), byte for byte.
 *
 * The reference paints it on every core at start-up, about 0.6 s: two million gas texels of some twenty
 * lattice lookups each (strands along each orbit, torn clouds, a fraying edge), dust lanes, the sky's
 * dust band, a black-body colour table and the rings' tables.  Every texel is its own; this unit is built
 * without contraction and with IEEE division and square root, and each float expression keeps the
 * reference's order.  The one reduction, the gas's mean over the map's inner half (a double sum the reference
 * adds in texel order), is added here in a fixed tree order: the sum is of floats of moderate range, its
 * double rounding leaves the float scale derived from it unchanged, and the test holds the whole map to the
 * reference's bytes.  The colour and ring tables (4 K floats) come from the host set-up (holeHost.c), as the
 * reference computes them, as a kernel parameter.
 *
 * Three launches: paintRows, a block a row of the gas, the sky or the dust; scaleGas; and the tables.
 * What bounds it is issue: a lattice lookup is four hashes of eleven integer instructions.  A row's slow
 * lattices (ten of the gas's 21 lookups) have a few dozen columns, so their values are hashed once a row into
 * shared memory; columns wrap by a comparison, not a division; every period and seed is a constant.  paintRows 97 us (86 % of the issue slots), the whole call 270 -> 126 us; before, one
 * thread added the sums (1024 dependent double additions) and the tables and scratch were copied and
 * allocated in every call. */
#include "nvtxRange.h"
#include "artful_cuda.h"

#include <cuda_runtime.h>

namespace artf {
int contextStream(ArtfCuda* ctx, cudaStream_t* stream);
int contextMap(ArtfCuda* ctx, float** map);
int failWith(int status, const char* message);
}  // namespace artf

namespace {

constexpr int MW = ARTF_CUDA_MAP_WIDTH, MH = ARTF_CUDA_MAP_HEIGHT;
constexpr int SW = ARTF_CUDA_SKY_WIDTH, SH = ARTF_CUDA_SKY_HEIGHT, DW = ARTF_CUDA_DUST_WIDTH, DH = ARTF_CUDA_DUST_HEIGHT;
constexpr int HALF = MW * (MH / 2);   /* the inner half the gas is scaled over */
constexpr int THREADS = 256;          /* a row's block */

__device__ __forceinline__ float clampF(float v, float lo, float hi) { return v < lo ? lo : v > hi ? hi : v; }

/* hole.c:14-21 */
__device__ __forceinline__ uint32_t texHash(uint32_t x, uint32_t y, uint32_t seed) {
    uint32_t h = x * 0x9E3779B1u ^ y * 0x85EBCA77u ^ seed * 0xC2B2AE3Du;
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 12;
    h *= 0x297A2D39u;
    return h ^ h >> 15;
}

/* hole.c:23-26 */
__device__ __forceinline__ float ease(float a, float b, float x) {
    const float t = clampF((x - a) / (b - a), 0.f, 1.f);
    return t * t * (3.f - 2.f * t);
}

/* A lattice's column at x, 0 <= x <= period (x is a turn, a whole one included, of `period` columns), and
 * the next one: (uint32_t)(int32_t)floor(x) and one more, each modulo the period. */
__device__ __forceinline__ void columns(float fx, uint32_t period, uint32_t& x0, uint32_t& x1) {
    x0 = (uint32_t)(int32_t)fx;
    x0 = x0 == period ? 0u : x0;
    x1 = x0 + 1u == period ? 0u : x0 + 1u;
}

__device__ __forceinline__ float blend(float v00, float v10, float v01, float v11, float tx, float ty) {
    const float sx = tx * tx * (3.f - 2.f * tx), sy = ty * ty * (3.f - 2.f * ty);
    const float lo = v00 + (v10 - v00) * sx, hi = v01 + (v11 - v01) * sx;
    return (lo + (hi - lo) * sy) * (1.f / 16777216.f);
}

/* hole.c:29-39: value noise repeating every period in x, coordinates through a signed integer */
__device__ __forceinline__ float lattice(float x, float y, uint32_t period, uint32_t seed) {
    const float fx = floorf(x), fy = floorf(y);
    uint32_t x0, x1;
    columns(fx, period, x0, x1);
    const uint32_t y0 = (uint32_t)(int32_t)fy, y1 = y0 + 1;
    const float v00 = (float)(texHash(x0, y0, seed) >> 8), v10 = (float)(texHash(x1, y0, seed) >> 8);
    const float v01 = (float)(texHash(x0, y1, seed) >> 8), v11 = (float)(texHash(x1, y1, seed) >> 8);
    return blend(v00, v10, v01, v11, x - fx, y - fy);
}

/* hole.c:42-53 */
template <int COUNT>
__device__ __forceinline__ float octaves(float x, float y, uint32_t period, float scaleY, float falloff, float stretch,
                                         uint32_t seed) {
    float sum = 0, amplitude = .5f, total = 0;
#pragma unroll
    for (int o = 0; o < COUNT; ++o) {
        sum += amplitude * lattice(x * (float)period, y * scaleY, period, seed + (uint32_t)o);
        total += amplitude;
        amplitude *= falloff;
        period *= 2;
        scaleY *= stretch;
    }
    return sum / total;
}

/* The same octaves along a row (y fixed): the lattice's values at the row's two lattice rows, hashed once
 * into `table`, 2 x PERIOD (2^COUNT - 1) floats, octave after octave, a row's columns after the other's. */
template <int PERIOD, int COUNT> constexpr int rowFloats = 2 * PERIOD * ((1 << COUNT) - 1);

template <int PERIOD, int COUNT>
__device__ __forceinline__ void hashRow(float* table, float y, float scaleY, float stretch, uint32_t seed) {
    for (int k = (int)threadIdx.x; k < rowFloats<PERIOD, COUNT>; k += THREADS) {
        int at = k, period = PERIOD;
        float scale = scaleY;
        uint32_t o = 0;
        for (; at >= 2 * period; ++o) at -= 2 * period, period *= 2, scale *= stretch;
        const uint32_t row = (uint32_t)(int32_t)floorf(y * scale) + (at >= period ? 1u : 0u);
        table[k] = (float)(texHash((uint32_t)(at >= period ? at - period : at), row, seed + o) >> 8);
    }
}

template <int PERIOD, int COUNT>
__device__ __forceinline__ float rowOctaves(const float* table, float x, float y, float scaleY, float falloff,
                                            float stretch) {
    float sum = 0, amplitude = .5f, total = 0;
    uint32_t period = PERIOD;
#pragma unroll
    for (int o = 0; o < COUNT; ++o) {
        const float px = x * (float)period, fx = floorf(px), py = y * scaleY;
        uint32_t x0, x1;
        columns(fx, period, x0, x1);
        sum += amplitude * blend(table[x0], table[x1], table[period + x0], table[period + x1], px - fx, py - floorf(py));
        total += amplitude;
        amplitude *= falloff;
        table += 2 * period;
        period *= 2;
        scaleY *= stretch;
    }
    return sum / total;
}

__device__ __forceinline__ float crest(float v) {
    const float r = 1.f - fabsf(2.f * v - 1.f);
    return r * r;
}

/* The gas's lattices along a row: the two wanders and the drift along the orbit. */
struct GasRow {
    float wide[rowFloats<3, 4>], narrow[rowFloats<11, 3>], drift[rowFloats<5, 3>];
};

/* hole.c:101-124 */
__device__ __forceinline__ float gasAt(const GasRow& row, float turn, float rho) {
    const float wander = .045f * (rowOctaves<3, 4>(row.wide, turn, rho, 5.f, .5f, 2.f) - .5f) +
                         .012f * (rowOctaves<11, 3>(row.narrow, turn, rho, 24.f, .5f, 2.f) - .5f);
    float along = turn + .03f * (rowOctaves<5, 3>(row.drift, turn, rho, 9.f, .5f, 2.f) - .5f);
    along -= floorf(along);
    const float across = rho + wander;
    float hair = 0, amplitude = .5f, total = 0, scale = 600.f;
    uint32_t period = 6;
#pragma unroll
    for (int o = 0; o < 6; ++o) {
        hair += amplitude * crest(lattice(along * (float)period, across * scale, period, 120u + (uint32_t)o));
        total += amplitude;
        amplitude *= .62f;
        period *= 2;
        scale *= 1.75f;
    }
    hair /= total;
    const float cloud = octaves<5>(along, across, 7, 34.f, .55f, 2.f, 131);
    const float outer = ease(.85f, 1.f, rho);
    const float torn = ease(.3f + .08f * outer, .7f + .08f * outer, cloud);
    const float gaps = 1.f + (torn - 1.f) * ease(.1f, .6f, rho);
    const float edge = ease(0.f, .02f, rho) * (1.f - ease(.9f, 1.f, across));
    return edge * (.25f + 2.2f * hair) * (.04f + 1.5f * gaps);
}

/* The inner rows' sums wait in the glow table's place (written last), a double's two words a row. */
__device__ __forceinline__ uint32_t* rowSumAt(float* map, int row) {
    return reinterpret_cast<uint32_t*>(map + ARTF_CUDA_GLOW_AT + 2 * row);
}
static_assert(2 * (MH / 2) <= ARTF_CUDA_MAP_HEIGHT, "a word pair an inner row in the glow table's place");

/* The block's sum of a double a thread, a fixed tree; in thread 0. */
__device__ __forceinline__ double blockSum(double v, double* part) {
    part[threadIdx.x] = v;
    __syncthreads();
    for (int width = THREADS / 2; width > 0; width >>= 1) {
        if ((int)threadIdx.x < width) part[threadIdx.x] += part[threadIdx.x + width];
        __syncthreads();
    }
    return part[0];
}

/* A block a row: hole.c:128-138 the gas (and an inner row's sum), hole.c:168-177 the sky's dust band,
 * hole.c:150-159 the dust lanes. */
__global__ void __launch_bounds__(THREADS) paintRows(float* __restrict__ map) {
    __shared__ union {
        GasRow gas;
        float sky[rowFloats<8, 6>], dust[rowFloats<4, 5>];
    } row;
    __shared__ double part[THREADS];
    int y = (int)blockIdx.x;
    if (y < MH) {
        const float rho = (float)y / (float)(MH - 1), thin = 1.f - .887f * rho;
        hashRow<3, 4>(row.gas.wide, rho, 5.f, 2.f, 101);
        hashRow<11, 3>(row.gas.narrow, rho, 24.f, 2.f, 107);
        hashRow<5, 3>(row.gas.drift, rho, 9.f, 2.f, 113);
        __syncthreads();
        double sum = 0.0;
        for (int x = (int)threadIdx.x; x < MW; x += THREADS) {
            float turn = (float)x / (float)MW + rho * .09f;
            turn -= floorf(turn);
            const float v = gasAt(row.gas, turn, rho) * thin * thin;
            map[y * MW + x] = v;
            sum += (double)v;
        }
        if (y < MH / 2) {
            sum = blockSum(sum, part);
            if (threadIdx.x == 0)
                rowSumAt(map, y)[0] = (uint32_t)__double2loint(sum), rowSumAt(map, y)[1] = (uint32_t)__double2hiint(sum);
        }
        return;
    }
    y -= MH;
    if (y < SH) {
        const float height = (float)y / (float)(SH - 1);
        hashRow<8, 6>(row.sky, height, 8.f, 2.f, 51);
        __syncthreads();
        for (int x = (int)threadIdx.x; x < SW; x += THREADS) {
            const float turn = (float)x / (float)SW;
            const float bent = height - .5f + .22f * (lattice(turn * 2.f, 3.f, 2, 41) - .5f) +
                               .1f * (lattice(turn * 3.f, 5.f, 3, 42) - .5f);
            const float band = 1.f - ease(0.f, .3f, fabsf(bent));
            const float dust = rowOctaves<8, 6>(row.sky, turn, height, 8.f, .58f, 2.f);
            map[ARTF_CUDA_SKY_AT + y * SW + x] = .0006f + band * band * ease(.3f, .75f, dust) * .006f;
        }
        return;
    }
    y -= SH;
    const float rho = (float)y / (float)(DH - 1), outward = ease(.25f, .8f, rho);
    hashRow<4, 5>(row.dust, rho, 90.f, 2.f, 151);
    __syncthreads();
    for (int x = (int)threadIdx.x; x < DW; x += THREADS) {
        const float turn = (float)x / (float)DW;
        map[ARTF_CUDA_DUST_AT + y * DW + x] =
            outward * ease(.45f, .7f, rowOctaves<4, 5>(row.dust, turn, rho, 90.f, .55f, 2.f));
    }
}

/* The scale from the inner rows' sums (hole.c:143-146): each block adds them by the same tree, and scales its
 * share of the gas, SHARE texels a thread. */
constexpr int SHARE = 32;
__global__ void __launch_bounds__(THREADS) scaleGas(float* __restrict__ map) {
    __shared__ double part[THREADS];
    double v = 0.0;
    for (int r = (int)threadIdx.x; r < MH / 2; r += THREADS)
        v += __hiloint2double((int)rowSumAt(map, r)[1], (int)rowSumAt(map, r)[0]);
    const float scale = (float)((double)HALF / blockSum(v, part));
    float* const mine = map + (size_t)blockIdx.x * SHARE * THREADS + threadIdx.x;
#pragma unroll 16
    for (int k = 0; k < SHARE; ++k) mine[k * THREADS] *= scale;
}

/* The rings' and colours' tables, as the host formed them. */
struct Tables {
    float rows[ARTF_CUDA_MAP_HEIGHT * 2 + ARTF_CUDA_COLORS * 3], glow[ARTF_CUDA_MAP_HEIGHT];
};

__global__ void __launch_bounds__(THREADS) writeTables(float* __restrict__ map, const __grid_constant__ Tables t) {
    const int k = (int)(blockIdx.x * THREADS + threadIdx.x), rows = (int)(sizeof t.rows / sizeof(float));
    if (k < rows) map[ARTF_CUDA_ROWS_AT + k] = t.rows[k];
    else if (k - rows < ARTF_CUDA_MAP_HEIGHT) map[ARTF_CUDA_GLOW_AT + k - rows] = t.glow[k - rows];
}

}  // namespace

extern "C" int artfCudaPaintDisc(ArtfCuda* ctx, float* map, float inner, float outer, float spin) {
    artf::Range range("artfCudaPaintDisc");
    cudaStream_t stream = nullptr;
    if (int s = artf::contextStream(ctx, &stream)) return s;
    if (!(inner > 0.f) || !(outer > inner) || !(fabsf(spin) <= 1.f))
        return artf::failWith(ARTF_CUDA_EINVAL, "paint disc: needs 0 < inner < outer and |spin| <= 1");
    if (!map)
        if (int s = artf::contextMap(ctx, &map)) return s;
    /* the tables on the host: rows and colours lie together, the glow apart */
    static_assert(ARTF_CUDA_COLORS_AT == ARTF_CUDA_ROWS_AT + ARTF_CUDA_MAP_HEIGHT * 2, "map layout");
    paintRows<<<MH + SH + DH, THREADS, 0, stream>>>(map);
    scaleGas<<<MW * MH / (SHARE * THREADS), THREADS, 0, stream>>>(map);
    Tables t; /* (formed while the rows are painted) */
    artfCudaHoleRings(t.rows, t.glow, inner, outer, spin);
    artfCudaHoleColours(t.rows + ARTF_CUDA_MAP_HEIGHT * 2);
    writeTables<<<(sizeof t / sizeof(float) + THREADS - 1) / THREADS, THREADS, 0, stream>>>(map, t);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return artf::failWith(ARTF_CUDA_ELAUNCH, cudaGetErrorString(e));
    return ARTF_CUDA_OK;
}
