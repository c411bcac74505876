/* artful_cuda — the disc's gas on the GPU: the reference's fluid step (src/scene/fluid.c), byte for byte.
 *
 * The model (fluid.c:1-23): isothermal compressible flow in the disc's plane on 256 rings of 1024 cells,
 * density S and the velocity's departure from a circular orbit (vr along the radius, w along the orbit),
 * Kerr's orbital and epicyclic frequencies; eddies stirred in at random; a FARGO-style shift of each ring
 * along itself by its own orbit.  The reference steps it on the CPU every frame and uploads the 1 MB
 * field; here it stays on the device, where the trace reads it.
 *
 * Same bytes: this unit is built without contraction and with IEEE division and square root, and each
 * float expression keeps the reference's order of operations.  The reference's cell loops are
 * independent within a pass (each pass reads one copy of the fields and writes the other), so one thread
 * a cell computes what it computes.  Two things are ordered: the eddies, which overlap: each cell takes
 * them in their order, and an eddy changes a cell by that cell's own values alone, so the cells need not
 * wait for one another; and each ring's mean density, a sum in cell order, which one thread a ring adds
 * up.  The random draws that place the eddies (a xorshift sequence) are made on the host, in the
 * reference's order, and travel with the launches as kernel parameters.
 *
 * Work layout: 7 fields of 256 x 1024 floats (7 MB, L2-resident), one allocation.  A step is one launch on
 * the context's stream, `gasStep`: a block a ring, in clusters of eight rings that exchange what a ring
 * needs of its neighbours through shared memory.  What bounds a step is latency: the sum in cell order (1024
 * dependent additions, 1.9 us), three reads in turn of fields that other SMs have just written, and one
 * launch waiting for the last.  One block working through the eddies, and a launch a pass, took 62 us a
 * step; a launch for the velocities and one for the rest of each ring 10.8, one launch 9.7, and with a cell's
 * two velocities side by side, read together, 9.0 (24 steps a call: 1486 -> 265 -> 241 -> 222 us; of that the
 * launches as dependent ones 387 -> 265).  Two blocks a SM are as many as a step has: cut for three, the blocks
 * crowd on fewer SMs and 24 steps take 284. */
#include "nvtxRange.h"
#include "artful_cuda.h"

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

namespace artf {
int contextStream(ArtfCuda* ctx, cudaStream_t* stream);
int contextFluid(ArtfCuda* ctx, float** fluid);
struct GasStore;
cudaError_t takeGas(ArtfCuda* ctx, size_t bytes, void** block, GasStore** store);
void giveGas(GasStore* store, void* block, bool idle);
int failWith(int status, const char* message);
}  // namespace artf

namespace {

constexpr int FW = ARTF_CUDA_FLUID_WIDTH;  /* cells around a ring */
constexpr int FH = ARTF_CUDA_FLUID_HEIGHT; /* rings */
constexpr float DT = .2f;                  /* fluid.c:28 */
#define ARC (6.2831853f / (float)FW)       /* fluid.c:29 */
constexpr int WARM_STEPS = 60;             /* fluid.c:31 */
constexpr float WOUND_TIME = 900.f;        /* fluid.c:32 */
constexpr int EDDIES_A_STEP = 16;          /* fluid.c:232-234: two large, fourteen small */
constexpr int START_EDDIES = 200;          /* fluid.c:312 */
constexpr int EDDIES_A_LAUNCH = 128;       /* a launch's room for them */
constexpr int RING_THREADS = 512;          /* a ring's block: two cells a thread */
constexpr int RINGS = 8;                   /* a cluster's rings */
constexpr int FIELD = FW * FH;

/* What a cell's passes take from its ring alone (fluid.c:98-106, 128-135, 155-165, 270-287), formed once on
 * the host in the reference's float operations (IEEE there and here: the same values; on the device each
 * cell formed them again with five divisions): its radius and its neighbours', orbital and epicyclic
 * terms, sound speed squared, the gradients' factors, the cubic its shift reads with, and the envelope
 * and fall-off of what shows. */
struct Ring {
    float radius, up, down, angular, epicyclic, sound2, toCells, toRows, invR, invSpan, invArc, keep, refill;
    float k0, k1, k2, k3, envelope, fall;
    int shift;
};

/* One eddy, placed and shaped on the host (fluid.c:188-201). */
struct Eddy {
    float r0, size, strength, clump, invSize2;
    int i0, reach;
};

__host__ __device__ __forceinline__ float clampF(float v, float lo, float hi) { return v < lo ? lo : v > hi ? hi : v; }
__host__ __device__ __forceinline__ float lesser(float a, float b) { return b < a ? b : a; }
__host__ __device__ __forceinline__ float greater(float a, float b) { return a < b ? b : a; }
__host__ __device__ __forceinline__ int atMost(int a, int b) { return a < b ? a : b; }
__host__ __device__ __forceinline__ int atLeast(int a, int b) { return a > b ? a : b; }

__host__ __device__ __forceinline__ float ease(float a, float b, float x) {
    const float t = clampF((x - a) / (b - a), 0.f, 1.f);
    return t * t * (3.f - 2.f * t);
}

__device__ __forceinline__ uint32_t cellHash(uint32_t x, uint32_t y, uint32_t seed) {
    uint32_t h = x * 0x9E3779B1u ^ y * 0x85EBCA77u ^ seed * 0xC2B2AE3Du;
    h = (h ^ h >> 15) * 0x2C1B3C6Du;
    h = (h ^ h >> 12) * 0x297A2D39u;
    return h ^ h >> 15;
}

/* fluid.c:71-80 */
__device__ __forceinline__ float noise(float x, float y, uint32_t period, uint32_t seed) {
    const float fx = floorf(x), fy = floorf(y), tx = x - fx, ty = y - fy;
    const uint32_t x0 = (uint32_t)fx & (period - 1), x1 = (x0 + 1) & (period - 1), y0 = (uint32_t)fy, y1 = y0 + 1;
    const float v00 = (float)(cellHash(x0, y0, seed) >> 8), v10 = (float)(cellHash(x1, y0, seed) >> 8);
    const float v01 = (float)(cellHash(x0, y1, seed) >> 8), v11 = (float)(cellHash(x1, y1, seed) >> 8);
    const float sx = tx * tx * (3.f - 2.f * tx), sy = ty * ty * (3.f - 2.f * ty);
    const float lo = v00 + (v10 - v00) * sx, hi = v01 + (v11 - v01) * sx;
    return (lo + (hi - lo) * sy) * (1.f / 16777216.f);
}

/* fluid.c:82-93, where it reads: the cell's two columns and two rows, and how far between them (an index
 * never leaves the field: y0 <= FH - 2, columns wrap). */
struct Between {
    uint32_t lo0, lo1; /* of the lower row; the upper's lie FW on */
    float px, py;
};
__device__ __forceinline__ Between betweenOf(float x, float y) {
    const float fy = clampF(y, 0.f, (float)(FH - 1) - .001f);
    const int y0 = (int)fy;
    const float fx = floorf(x);
    const uint32_t x0 = (uint32_t)(int)fx & (FW - 1), row = (uint32_t)y0 * FW;
    return {row + x0, row + ((x0 + 1) & (FW - 1)), x - fx, fy - (float)y0};
}
__device__ __forceinline__ float bilinear(const Between& b, float lo0, float lo1, float hi0, float hi1) {
    const float top = lo0 + (lo1 - lo0) * b.px, bottom = hi0 + (hi1 - hi0) * b.px;
    return top + (bottom - top) * b.py;
}

/* ---- kernels: one thread a cell, unless said otherwise ------------------------------------------ */

/* fluid.c:291-311: the start, clumps the shear has long been drawing out */
__global__ void __launch_bounds__(256) seedDensity(float* __restrict__ s, const Ring* __restrict__ rings) {
    const int cell = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (cell >= FIELD) return;
    const int j = cell / FW, i = cell - j * FW;
    const float rho = (float)j / (float)(FH - 1), wound = rings[j].angular * WOUND_TIME / 6.2831853f;
    float turn = (float)i / (float)FW - wound;
    turn -= floorf(turn);
    float sum = 0, amplitude = .5f, total = 0, across = 14.f;
    uint32_t period = 16;
    for (uint32_t o = 0; o < 5; ++o) {
        sum += amplitude * noise(turn * (float)period, rho * across, period, 7 + o);
        total += amplitude;
        amplitude *= .72f;
        period *= 2;
        across *= 2.f;
    }
    const float v = sum / total;
    s[cell] = .06f + 3.4f * ease(.34f, .68f, v) * ease(.34f, .68f, v);
}

/* A launch's eddies, in their order, as a kernel parameter: a step's 16, or 128 (3.6 KB, under the 4 KB
 * every driver takes) of a gas's start. */
template <int N> struct Eddies {
    int count;
    Eddy e[N];
};

/* The launches of a run follow one another at once (programmatic dependent launch): a kernel may start
 * while the one before it drains, fetches what no kernel writes, and waits here, before its first read of
 * the fields, until that one has finished and its writes are visible.  The fields' pointers are not
 * __restrict__: their reads stay below the wait. */
__device__ __forceinline__ void startNext() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void waitBefore() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

/* How strongly an eddy's shape reaches the cell (ring radius r, column i), fluid.c:202-214: whether it does,
 * and there its shape and the offsets from its middle.  Columns -reach .. reach: fewer than FW, so a cell
 * is at one offset at most. */
__device__ __forceinline__ bool eddyAt(const Eddy& q, float r, int i, float& shape, float& dr, float& dx) {
    dr = r - q.r0;
    if (dr * dr > 6.25f * q.size * q.size) return false;
    const int di = ((i - q.i0 + FW / 2) & (FW - 1)) - FW / 2;
    if (di > q.reach || di < -q.reach) return false;
    dx = (float)di * r * ARC;
    const float d2 = (dr * dr + dx * dx) * q.invSize2;
    if (d2 > 6.25f) return false;
    const float g = 1.f - d2 * .16f;
    shape = g * g * g;
    return true;
}

/* What an eddy does to a cell it reaches (fluid.c:215-217): to its velocities, and to its density. */
__device__ __forceinline__ void stirFlow(const Eddy& q, float r, int i, float2& v) {
    float shape, dr, dx;
    if (!eddyAt(q, r, i, shape, dr, dx)) return;
    v.x -= q.strength * shape * dx / q.size;
    v.y += q.strength * shape * dr / q.size;
}

__device__ __forceinline__ void stirDensity(const Eddy& q, float r, int i, float& s) {
    float shape, dr, dx;
    if (eddyAt(q, r, i, shape, dr, dx)) s = clampF(s * (1.f + q.clump * shape), .03f, 8.f);
}

/* Eddies on their own (a gas's start, and its first step's): a block a ring, so that an eddy out of the
 * ring's reach costs the block one uniform test. */
__global__ void __launch_bounds__(RING_THREADS) stir(float* s, float2* flow, const Ring* __restrict__ rings,
                                                     const __grid_constant__ Eddies<EDDIES_A_LAUNCH> eddies) {
    const int j = (int)blockIdx.x;
    const float r = rings[j].radius;
    startNext();
    waitBefore();
    for (int i = (int)threadIdx.x; i < FW; i += RING_THREADS) {
        const uint32_t at = (uint32_t)(j * FW + i);
        float cellS = s[at];
        float2 v = flow[at];
        for (int e = 0; e < eddies.count; ++e) {
            stirFlow(eddies.e[e], r, i, v);
            stirDensity(eddies.e[e], r, i, cellS);
        }
        s[at] = cellS, flow[at] = v;
    }
}

/* fluid.c:96-124: a cell's new velocities (along the radius, along the orbit) */
__device__ __forceinline__ float2 velocitiesAt(const float* s, const float2* flow, const Ring& g, int j, int i) {
    const uint32_t row = (uint32_t)(j * FW), cell = row + (uint32_t)i;
    const uint32_t up = j < FH - 1 ? cell + FW : cell, down = j > 0 ? cell - FW : cell;
    const float2 v = flow[cell];
    const Between b = betweenOf((float)i - v.y * g.toCells, (float)j - v.x * g.toRows);
    const float2 lo0 = flow[b.lo0], lo1 = flow[b.lo1], hi0 = flow[b.lo0 + FW], hi1 = flow[b.lo1 + FW];
    const float v0 = bilinear(b, lo0.x, lo1.x, hi0.x, hi1.x), w0 = bilinear(b, lo0.y, lo1.y, hi0.y, hi1.y);
    const float inv = 1.f / s[cell];
    const float gradR = (s[up] - s[down]) * g.invSpan * inv;
    const float gradPhi = (s[row + ((i + 1) & (FW - 1))] - s[row + ((i - 1) & (FW - 1))]) * g.invArc * inv;
    const float w1 = w0 + DT * (-g.epicyclic * v0 - v0 * w0 * g.invR - g.sound2 * gradPhi);
    const float v1 = v0 + DT * (2.f * g.angular * w1 + w1 * w1 * g.invR - g.sound2 * gradR);
    return make_float2(clampF(v1 * g.keep, -.4f, .4f), clampF(w1 * g.keep, -.4f, .4f));
}

/* fluid.c:126-151: a cell's new density, from the old ones and the new velocities: its ring's, and the radial
 * ones of the rings above and below at its column. */
__device__ __forceinline__ float densityAt(const float* s, const float2* flow, float vrUp, float vrDown, const Ring& g, int j,
                                           int i) {
    const float drift = -.004f;
    const float2 v = flow[i];
    const Between b = betweenOf((float)i - v.y * g.toCells, (float)j - (v.x + drift) * g.toRows);
    const float moved = bilinear(b, s[b.lo0], s[b.lo1], s[b.lo0 + FW], s[b.lo1 + FW]);
    const float spread = (g.up * vrUp - g.down * vrDown) * g.invSpan * g.invR +
                         (flow[(i + 1) & (FW - 1)].y - flow[(i - 1) & (FW - 1)].y) * g.invArc;
    const float next = moved * (1.f - DT * clampF(spread, -2.f, 2.f));
    return clampF(next + (1.f - next) * g.refill, .03f, 8.f);
}

/* fluid.c:153-173: a ring moved along itself by its orbit, a Catmull-Rom cubic held within its two middle
 * neighbours */
__device__ __forceinline__ float slide(float p0, float p1, float p2, float p3, const Ring& g) {
    return clampF(g.k0 * p0 + g.k1 * p1 + g.k2 * p2 + g.k3 * p3, lesser(p1, p2), greater(p1, p2));
}
__device__ __forceinline__ float slideCell(const float* in, int i, const Ring& g) {
    const int at = i + g.shift;
    return slide(in[(at - 1) & (FW - 1)], in[at & (FW - 1)], in[(at + 1) & (FW - 1)], in[(at + 2) & (FW - 1)], g);
}
__device__ __forceinline__ float2 slideCell(const float2* in, int i, const Ring& g) {
    const int at = i + g.shift;
    const float2 p0 = in[(at - 1) & (FW - 1)], p1 = in[at & (FW - 1)], p2 = in[(at + 1) & (FW - 1)], p3 = in[(at + 2) & (FW - 1)];
    return make_float2(slide(p0.x, p1.x, p2.x, p3.x, g), slide(p0.y, p1.y, p2.y, p3.y, g));
}

/* A step: a block a ring, clusters of RINGS neighbouring rings.  Each block finds its ring's new velocities
 * from the old fields; the new densities take the neighbours' radial ones, which the cluster's blocks read
 * from one another's shared memory (the rings the cluster borders on are found by all its blocks, a share
 * each); the rest stays within the ring: the shift of the three fields along it, the mean drawn to 1
 * (fluid.c:221-229: a sum in cell order, by one thread of a warp of its own, while the others stir the
 * velocities), the next step's eddies, and, when `field` is given, what shows of the ring
 * (fluid.c:175-186).  The fields are read from one copy and written to the other. */
__global__ void __cluster_dims__(RINGS, 1, 1) __launch_bounds__(RING_THREADS + 32)
    gasStep(const float* s, const float2* flow, float* outS, float2* outFlow, const Ring* __restrict__ rings,
            float* field, const __grid_constant__ Eddies<EDDIES_A_STEP> eddies) {
    constexpr int CELLS = FW / RING_THREADS, SHARE = FW / RINGS;
    __shared__ __align__(16) float slidRing[FW];
    __shared__ float ringS[FW];
    __shared__ float2 ringFlow[FW];
    __shared__ float outer[FW];   /* the radial velocities of the ring beyond, in the first and last block */
    __shared__ uint32_t reaching; /* the eddies that reach the ring at all, a bit each */
    __shared__ float scale;
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int tid = (int)threadIdx.x, j = (int)blockIdx.x, rank = j % RINGS;
    const bool helper = tid >= RING_THREADS;
    /* (this block has started: the others hear of it, and wait for it, before they write to its shared memory; the
     * step before hides it: as fast without, where a block's memory read after the next barrier takes 224 us) */
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const Ring g = rings[j];
    const uint32_t row = (uint32_t)(j * FW);
    if (helper) {
        const int e = tid - RING_THREADS;
        const float dr = e < eddies.count ? g.radius - eddies.e[e & (EDDIES_A_STEP - 1)].r0 : 0.f;
        const float size = eddies.e[e & (EDDIES_A_STEP - 1)].size;
        const uint32_t bits = __ballot_sync(0xFFFFFFFFu, e < eddies.count && !(dr * dr > 6.25f * size * size));
        if (e == 0) reaching = bits;
    }
    waitBefore();
    if (!helper) {
#pragma unroll
        for (int c = 0; c < CELLS; ++c) {
            const int i = tid + c * RING_THREADS;
            ringFlow[i] = velocitiesAt(s, flow, g, j, i);
        }
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (!helper) {
        /* this block's share of the rings below and above the cluster, where there are any (found whole by the
         * outer blocks they cost 1.3 us a step) */
        if (tid < 2 * SHARE) {
            const bool below = tid < SHARE;
            const int beyond = j - rank + (below ? -1 : RINGS), i = rank * SHARE + (below ? tid : tid - SHARE);
            if (beyond >= 0 && beyond < FH)
                cluster.map_shared_rank(outer, below ? 0 : RINGS - 1)[i] = velocitiesAt(s, flow, rings[beyond], beyond, i).x;
        }
    }
    cluster.sync();
    startNext(); /* (any later is alike; at the kernel's start its blocks are in the way of these: 225, not 222 us) */
    if (!helper) {
        /* (the first and last ring border on themselves) */
        const bool outBelow = rank == 0 && j > 0, outAbove = rank == RINGS - 1 && j < FH - 1;
        const float* below = outBelow ? outer : &cluster.map_shared_rank(ringFlow, rank > 0 ? rank - 1 : rank)->x;
        const float* above = outAbove ? outer : &cluster.map_shared_rank(ringFlow, rank < RINGS - 1 ? rank + 1 : rank)->x;
        const int stepBelow = outBelow ? 1 : 2, stepAbove = outAbove ? 1 : 2;
#pragma unroll
        for (int c = 0; c < CELLS; ++c) {
            const int i = tid + c * RING_THREADS;
            ringS[i] = densityAt(s, ringFlow, above[i * stepAbove], below[i * stepBelow], g, j, i);
        }
    }
    __syncthreads();
    /* (no block leaves while a neighbour may read its ring: waited for at the end; nothing is handed over) */
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    float slidS[CELLS];
    if (!helper) {
#pragma unroll
        for (int c = 0; c < CELLS; ++c)
            slidRing[tid + c * RING_THREADS] = slidS[c] = slideCell(ringS, tid + c * RING_THREADS, g);
    }
    __syncthreads();
    if (helper) {
        if (tid == RING_THREADS) {
            float sum = 0;
            const float4* four = reinterpret_cast<const float4*>(slidRing);
#pragma unroll 32
            for (int i = 0; i < FW / 4; ++i) {
                const float4 q = four[i];
                sum += q.x;
                sum += q.y;
                sum += q.z;
                sum += q.w;
            }
            const float mean = sum * (1.f / (float)FW);
            scale = 1.f + .03f * (1.f / mean - 1.f);
        }
        __syncthreads();
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        return;
    }
    /* The eddies near each cell: of the 16 some four reach a ring, and each a few dozen of its 1024 columns,
     * so most cells are done with a test of columns an eddy. */
    uint32_t near[CELLS];
#pragma unroll
    for (int c = 0; c < CELLS; ++c) {
        const int i = tid + c * RING_THREADS;
        float2 v = slideCell(ringFlow, i, g);
        near[c] = 0;
        for (uint32_t bits = reaching; bits; bits &= bits - 1) {
            const Eddy& q = eddies.e[__ffs((int)bits) - 1];
            if (((i - q.i0 + q.reach) & (FW - 1)) <= 2 * q.reach) near[c] |= bits & (0u - bits);
        }
        for (uint32_t bits = near[c]; bits; bits &= bits - 1)
            stirFlow(eddies.e[__ffs((int)bits) - 1], g.radius, i, v);
        outFlow[row + i] = v;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < CELLS; ++c) {
        const int i = tid + c * RING_THREADS;
        float v = clampF(slidS[c] * scale, .03f, 8.f);
        if (field) {
            const float shown = v * g.envelope;
            field[row + i] = g.fall * ease(.1f, 1.1f, shown) * lesser(shown, 2.2f);
        }
        for (uint32_t bits = near[c]; bits; bits &= bits - 1)
            stirDensity(eddies.e[__ffs((int)bits) - 1], g.radius, i, v);
        outS[row + i] = v;
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace

struct ArtfCudaFluid {
    ArtfCuda* ctx;
    int device;
    cudaStream_t stream;
    float inner, outer;
    float* block;          /* the seven fields and the rings' terms, one allocation */
    artf::GasStore* store; /* where it goes back to */
    float* dens[2];
    float2* flow[2];       /* velocities along the radius and the orbit, side by side: read together */
    float* field;
    int cur;               /* which copy of the three fields is the current one */
    Ring* rings;           /* device copy */
    Ring host[FH];
    uint32_t state;        /* fluid.c:49 xorshift32 */
    double time;
};

namespace {

constexpr size_t GAS_BYTES = sizeof(float) * FIELD * 7 + sizeof(Ring) * FH;

/* A gas's memory given back, once the device is done with it (work on other streams that reads the field among
 * it). */
void giveGas(ArtfCudaFluid* f) {
    if (!f->block) return;
    int current = 0;
    const bool known = cudaGetDevice(&current) == cudaSuccess;
    cudaSetDevice(f->device);
    const bool idle = cudaDeviceSynchronize() == cudaSuccess;
    artf::giveGas(f->store, f->block, idle);
    if (known) cudaSetDevice(current);
}

uint32_t draw(ArtfCudaFluid* f) {
    uint32_t x = f->state;
    x ^= x << 13;
    x ^= x >> 17;
    x ^= x << 5;
    f->state = x;
    return x;
}
float uniform(ArtfCudaFluid* f) { return (float)(draw(f) >> 8) * (1.f / 16777216.f); }

/* fluid.c:188-201: where an eddy goes and its shape, with the reference's draws in its order */
Eddy placeEddy(ArtfCudaFluid* f, bool small) {
    Eddy q;
    const float u = uniform(f);
    q.r0 = f->inner + (f->outer - f->inner) * u * u;
    int j0 = 0; /* the first ring at or past r0, or the last (the rings' radii ascend) */
    for (int past = FH - 1; j0 < past;) {
        const int mid = (j0 + past) / 2;
        if (f->host[mid].radius < q.r0) j0 = mid + 1;
        else past = mid;
    }
    q.i0 = (int)(draw(f) & (FW - 1));
    q.size = q.r0 * (small ? .006f + .02f * uniform(f) : .02f + .1f * uniform(f));
    const float c = sqrtf(f->host[j0].sound2);
    q.strength = 0.f;
    if (!small) {
        const float sign = uniform(f) < .5f ? -1.f : 1.f;
        q.strength = sign * c * (.3f + .7f * uniform(f));
    }
    q.clump = (uniform(f) - .42f) * (small ? 1.5f : .5f);
    q.invSize2 = 1.f / (q.size * q.size);
    q.reach = atMost((int)(2.5f * q.size / (q.r0 * ARC)) + 1, FW / 2 - 1);
    return q;
}

/* The next `large` large and `small` small eddies, drawn in that order, after those q holds. */
template <int N> void drawEddies(ArtfCudaFluid* f, Eddies<N>& q, int large, int small) {
    for (int e = 0; e < large; ++e) q.e[q.count++] = placeEddy(f, false);
    for (int e = 0; e < small; ++e) q.e[q.count++] = placeEddy(f, true);
}

/* A kernel that may start while the stream's work before it drains, for those that wait in waitBefore. */
template <typename... P, typename... A>
cudaError_t follow(ArtfCudaFluid* f, void (*kernel)(P...), unsigned blocks, unsigned threads, const A&... args) {
    cudaLaunchAttribute early;
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(blocks), c.blockDim = dim3(threads), c.stream = f->stream, c.attrs = &early, c.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, kernel, P(args)...);
    if (e != cudaSuccess) (void)cudaGetLastError(); /* (or the next launch's check would report it) */
    return e;
}

static_assert(START_EDDIES % EDDIES_A_LAUNCH + EDDIES_A_STEP <= EDDIES_A_LAUNCH, "the last launch holds both");

/* A gas's start: its eddies (fluid.c:309-313), and its first step's. */
int stirStart(ArtfCudaFluid* f) {
    Eddies<EDDIES_A_LAUNCH> q;
    cudaError_t e = cudaSuccess;
    for (int left = START_EDDIES; left >= 0 && e == cudaSuccess; left -= EDDIES_A_LAUNCH) {
        q.count = 0;
        drawEddies(f, q, atMost(left, EDDIES_A_LAUNCH), 0);
        if (left < EDDIES_A_LAUNCH) drawEddies(f, q, 2, EDDIES_A_STEP - 2);
        e = follow(f, stir, FH, RING_THREADS, f->dens[f->cur], f->flow[f->cur], f->rings, q);
    }
    if (e != cudaSuccess) return artf::failWith(ARTF_CUDA_ELAUNCH, cudaGetErrorString(e));
    return ARTF_CUDA_OK;
}

/* `steps` steps, one at least (fluid.c:231-241), and the field after them.  Between calls the fields stand
 * stirred for the step to come: each step's launch ends with the next one's eddies, which reach nothing that
 * shows. */
int advanceSteps(ArtfCudaFluid* f, int64_t steps) {
    Eddies<EDDIES_A_STEP> q;
    cudaError_t e = cudaSuccess;
    for (int64_t k = 0; k < steps && e == cudaSuccess; ++k) {
        const int from = f->cur, to = f->cur ^ 1;
        q.count = 0;
        drawEddies(f, q, 2, EDDIES_A_STEP - 2);
        e = follow(f, gasStep, FH, RING_THREADS + 32, f->dens[from], f->flow[from], f->dens[to], f->flow[to],
                   f->rings, k == steps - 1 ? f->field : (float*)nullptr, q);
        f->cur = to;
    }
    if (e != cudaSuccess) return artf::failWith(ARTF_CUDA_ELAUNCH, cudaGetErrorString(e));
    return ARTF_CUDA_OK;
}

}  // namespace

extern "C" void artfCudaFluidFree(ArtfCudaFluid* f) {
    if (!f) return;
    giveGas(f);
    free(f);
}

extern "C" int artfCudaFluidNew(ArtfCuda* ctx, float inner, float outer, float spin, double time,
                                ArtfCudaFluid** out) {
    artf::Range range("artfCudaFluidNew");
    if (!out) return artf::failWith(ARTF_CUDA_EINVAL, "out is NULL");
    *out = nullptr;
    if (!(inner > 0.f) || !(outer > inner) || !(fabsf(spin) <= 1.f) || !isfinite(time))
        return artf::failWith(ARTF_CUDA_EINVAL, "fluid: a disc needs 0 < inner < outer and |spin| <= 1");
    cudaStream_t stream = nullptr;
    if (int s = artf::contextStream(ctx, &stream)) return s;
    ArtfCudaFluid* f = (ArtfCudaFluid*)calloc(1, sizeof(ArtfCudaFluid));
    if (!f) return artf::failWith(ARTF_CUDA_ENOMEM, "host allocation");
    f->ctx = ctx, f->stream = stream, f->inner = inner, f->outer = outer;
    f->state = 0x9E3779B9u, f->time = time;
    if (cudaGetDevice(&f->device) != cudaSuccess ||
        artf::takeGas(ctx, GAS_BYTES, (void**)&f->block, &f->store) != cudaSuccess) {
        artfCudaFluidFree(f);
        return artf::failWith(ARTF_CUDA_ENOMEM, "fluid: device allocation");
    }
    for (int k = 0; k < 2; ++k)
        f->dens[k] = f->block + FIELD * (3 * k), f->flow[k] = (float2*)(f->block + FIELD * (3 * k + 1));
    f->field = f->block + FIELD * 6;
    f->rings = (Ring*)(f->block + FIELD * 7);
    /* the rings (fluid.c:270-290), on the host in float as the reference has them */
    const float k = 1.f - inner / outer;
    for (int j = 0; j < FH; ++j) {
        Ring& g = f->host[j];
        const float rho = (float)j / (float)(FH - 1), r = inner / (1.f - rho * k);
        g.radius = r;
        const float root = sqrtf(r), om = 1.f / (r * root + spin);
        g.angular = om;
        const float kappa2 = om * om * (1.f - 6.f / r + 8.f * spin / (r * root) - 3.f * spin * spin / (r * r));
        g.epicyclic = greater(kappa2, -.5f * om * om) / (2.f * om);
        const float c = .03f * r * om;
        g.sound2 = c * c;
        g.toCells = DT / (r * ARC), g.invR = 1.f / r, g.invArc = 1.f / (2.f * r * ARC);
        g.keep = 1.f - DT * .04f * om, g.refill = DT * .002f * om;
        const float cells = om * DT / ARC, whole = floorf(cells), t = 1.f - (cells - whole), t2 = t * t, t3 = t2 * t;
        g.shift = -(int)whole - 1;
        g.k0 = -.5f * t + t2 - .5f * t3, g.k1 = 1.f - 2.5f * t2 + 1.5f * t3;
        g.k2 = .5f * t + 2.f * t2 - 1.5f * t3, g.k3 = -.5f * t2 + .5f * t3;
        g.envelope = ease(inner + .5f, inner + 2.2f, r) * (1.f - .86f * ease(outer * .12f, outer * .8f, r));
        g.fall = sqrtf(inner / r);
    }
    for (int j = 0; j < FH; ++j) {
        Ring& g = f->host[j];
        g.up = f->host[atMost(j + 1, FH - 1)].radius, g.down = f->host[atLeast(j - 1, 0)].radius;
        g.invSpan = 1.f / (g.up - g.down);
        g.toRows = DT / ((g.up - g.down) * (j == 0 || j == FH - 1 ? 1.f : .5f));
    }
    cudaError_t e = cudaMemcpyAsync(f->rings, f->host, sizeof f->host, cudaMemcpyHostToDevice, stream);
    /* (at rest; the rest is written before it is read) */
    if (e == cudaSuccess) e = cudaMemsetAsync(f->flow[0], 0, sizeof(float2) * FIELD, stream);
    if (e == cudaSuccess) {
        seedDensity<<<(FIELD + 255) / 256, 256, 0, stream>>>(f->dens[0], f->rings);
        e = cudaGetLastError();
    }
    int status = e == cudaSuccess ? stirStart(f) : artf::failWith(ARTF_CUDA_ELAUNCH, cudaGetErrorString(e));
    if (!status) status = advanceSteps(f, WARM_STEPS);
    /* (the gas is there for any stream when the call returns) */
    if (!status && (e = cudaStreamSynchronize(stream)) != cudaSuccess)
        status = artf::failWith(ARTF_CUDA_ELAUNCH, cudaGetErrorString(e));
    if (status) {
        artfCudaFluidFree(f);
        return status;
    }
    f->time = time;
    *out = f;
    return ARTF_CUDA_OK;
}

extern "C" int artfCudaFluidAdvance(ArtfCudaFluid* f, double time, int* stepped) {
    artf::Range range("artfCudaFluidAdvance");
    if (stepped) *stepped = 0;
    if (!f || !isfinite(time)) return artf::failWith(ARTF_CUDA_EINVAL, "no fluid, or a time that is not finite");
    cudaStream_t stream = nullptr;
    if (int s = artf::contextStream(f->ctx, &stream)) return s;
    double clock = f->time;
    const int steps = artfCudaFluidClock(&clock, time);
    if (steps > 0)
        if (int s = advanceSteps(f, steps)) return s;
    f->time = clock;
    if (stepped) *stepped = steps > 0;
    return ARTF_CUDA_OK;
}

extern "C" int artfCudaFluidStep(ArtfCudaFluid* f, int64_t steps, double time) {
    artf::Range range("artfCudaFluidStep");
    if (!f || steps < 0 || !isfinite(time)) return artf::failWith(ARTF_CUDA_EINVAL, "fluid step: no fluid, or bad steps or time");
    cudaStream_t stream = nullptr;
    if (int s = artf::contextStream(f->ctx, &stream)) return s;
    if (steps > 0)
        if (int s = advanceSteps(f, steps)) return s;
    f->time = time;
    return ARTF_CUDA_OK;
}

extern "C" int artfCudaUseFluid(ArtfCuda* ctx, const ArtfCudaFluid* f) {
    if (!f || f->ctx != ctx) return artf::failWith(ARTF_CUDA_EINVAL, "use fluid: no fluid, or one of another context");
    float* dst = nullptr;
    if (int s = artf::contextFluid(ctx, &dst)) return s;
    const cudaError_t e = cudaMemcpyAsync(dst, f->field, sizeof(float) * FIELD, cudaMemcpyDeviceToDevice, f->stream);
    if (e != cudaSuccess) return artf::failWith(ARTF_CUDA_ELAUNCH, cudaGetErrorString(e));
    return ARTF_CUDA_OK;
}

extern "C" const float* artfCudaFluidField(const ArtfCudaFluid* f) { return f ? f->field : nullptr; }
extern "C" double artfCudaFluidTime(const ArtfCudaFluid* f) { return f ? f->time : 0.0; }

extern "C" int artfCudaFluidRead(const ArtfCudaFluid* f, float* host) {
    if (!f || !host) return artf::failWith(ARTF_CUDA_EINVAL, "no fluid or no buffer");
    cudaError_t e = cudaMemcpyAsync(host, f->field, sizeof(float) * FIELD, cudaMemcpyDeviceToHost, f->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(f->stream);
    if (e != cudaSuccess) return artf::failWith(ARTF_CUDA_ELAUNCH, cudaGetErrorString(e));
    return ARTF_CUDA_OK;
}
