/* The C ABI's host code (abi.cu, no kernel in it) over a fake CUDA runtime whose device memory is the host's:
 * what the entry points hand to the launches and what they leave behind when one fails, without a GPU. */
#include "artful_cuda.h"
#include "lensLaunch.h"
#include "lensMixed.h"
#include "lensTangent.h"

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <set>
#include <vector>

static int failures = 0;
static void check(bool ok, const char* what) {
    if (!ok) ++failures, printf("failed: %s\n", what);
}

/* ---- the fake runtime ---------------------------------------------------------------------------- */

static cudaMemoryType pointerKind = cudaMemoryTypeUnregistered;
static bool hostPages = true;
static int launches = 0, pendingLaunches = 0; /* in all; and since the stream was last waited for */
static int failLaunch = -1;                   /* this one (from 0) fails */
static int events = 0, failEvent = -1;        /* event records of a call; the one (from 0) that fails */
static std::vector<float*> frames;            /* where each launch was to write its frame */
static bool failMalloc = false;
static std::set<void*> live;                  /* device allocations */

static cudaError_t launched(float4* hdr) {
    if (launches++ == failLaunch) return cudaErrorLaunchOutOfResources;
    frames.push_back((float*)hdr);
    ++pendingLaunches;
    return cudaSuccess;
}

extern "C" {
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.f, cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return events++ == failEvent ? cudaErrorInvalidValue : cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t bytes) {
    if (failMalloc) return cudaErrorMemoryAllocation;
    *p = aligned_alloc(256, (bytes + 255) / 256 * 256);
    live.insert(*p);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (p) check(live.erase(p) == 1, "memory freed that is not held");
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t bytes) { return *p = malloc(bytes), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaGetDevice(int* device) { return *device = 0, cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
#undef cudaGetDeviceProperties
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    memset(p, 0, sizeof *p);
    p->major = 10, p->minor = 3, p->multiProcessorCount = 152;
    p->pageableMemoryAccess = p->pageableMemoryAccessUsesHostPageTables = hostPages;
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, cudaMemcpyKind, cudaStream_t) {
    return memcpy(to, from, bytes), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t bytes, cudaStream_t) { return memset(p, v, bytes), cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    memset(a, 0, sizeof *a);
    a->type = pointerKind;
    a->hostPointer = (void*)p;
    a->devicePointer = pointerKind == cudaMemoryTypeUnregistered ? nullptr : (void*)p;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return pendingLaunches = 0, cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)1, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return pendingLaunches = 0, cudaSuccess; }

int artfCudaPostLaunch(const ArtfCudaHoleFrame*, const float*, float* const*, uint32_t*, void*) { return ARTF_CUDA_OK; }
}

/* ---- the launches -------------------------------------------------------------------------------- */

namespace artf {
cudaError_t launchExact(const TraceLaunch& l) { return launched(l.hdr); }
cudaError_t launchFast(const TraceLaunch& l) { return launched(l.hdr); }
cudaError_t launchFp64(const TraceLaunch& l) { return launched(l.hdr); }
size_t mixedViewBytes() { return 64; }
int mixedFillView(const TraceLaunch&, const ArtfCudaHoleFrame& f, const ArtfCudaHoleFrame64&, const float*, const float*,
                  float4* hdr, ArtfCudaRayEnd*, float4*, int, int, void* slot, int* tiles) {
    memcpy(slot, &hdr, sizeof hdr);
    *tiles = (int)((f.size[0] + 7) / 8 * ((f.size[1] + 3) / 4));
    return *tiles * 32;
}
size_t mixedOrderBytes(int tiles, int) { return (size_t)tiles * 8 + 64; }
cudaError_t launchMixedTable(const TraceLaunch&, const void*, int, int, size_t, int, void*, const void* view) {
    float4* hdr;
    memcpy(&hdr, view, sizeof hdr);
    return launched(hdr);
}
int adjointTiles(int, int) { return 1; }
size_t adjointViewBytes() { return 64; }
size_t adjointOrderBytes(int, int, int) { return 64; }
size_t adjointTrailBytes(int, int, int, int) { return 64; }
void adjointFillView(void*, const ArtfCudaHoleFrame&, const double*, double, const float*, const float*, const float*,
                     float*, float*) {}
cudaError_t launchAdjoint(const void*, int, int, int, int, unsigned long long*, float*, double*, cudaStream_t, void*,
                          void*) {
    return cudaSuccess;
}
cudaError_t launchTangents(const TraceLaunch&, const double*, double, double*) { return cudaSuccess; }

/* (the gas's side of its memory: abi.cu) */
struct GasStore;
cudaError_t takeGas(ArtfCuda* ctx, size_t bytes, void** block, GasStore** store);
void giveGas(GasStore* store, void* block, bool idle);
}  // namespace artf

/* ---- the checks ---------------------------------------------------------------------------------- */

static ArtfCuda* ctx;
static float* inputs;

static int render(int precision, float* out, uint32_t width, uint32_t height, int64_t bandRays) {
    ArtfCudaHoleFrame f;
    memset(&f, 0, sizeof f);
    f.size[0] = width, f.size[1] = height, f.size[2] = 1, f.size[3] = 1;
    ArtfCudaTraceOptions o;
    memset(&o, 0, sizeof o);
    o.precision = precision, o.bandRays = bandRays;
    frames.clear();
    launches = pendingLaunches = events = 0;
    return artfCudaHoleRender(ctx, &f, nullptr, inputs, 0, inputs, 0, &o, out, nullptr);
}

/* A host frame's address reaches the kernels, which store float4, only where it is aligned so. */
static void hostFrames() {
    const int precisions[] = {ARTF_CUDA_EXACT, ARTF_CUDA_MIXED};
    float* buffer = (float*)aligned_alloc(64, sizeof(float) * 4 * 17 * 16);
    for (int k = 0; k < 2; ++k) {
        pointerKind = k ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
        for (int p : precisions)
            for (int offset = 0; offset < 8; ++offset) {
                check(render(p, buffer + offset, 16, 16, 0) == ARTF_CUDA_OK && frames.size() == 1, "a host frame");
                check((uintptr_t)frames[0] % sizeof(float4) == 0, "a misaligned host frame handed to the kernels");
                check((frames[0] == buffer + offset) == (offset % 4 == 0), "an aligned host frame written directly");
                check(pendingLaunches == 0, "the call is synchronous");
            }
    }
    free(buffer);
}

/* A call that fails leaves none of its kernels in flight, with the caller's buffer: at the launch of a band, and
 * after the trace's launch, at the event behind it. */
static void failedCalls() {
    float* buffer = (float*)aligned_alloc(64, sizeof(float) * 4 * 16 * 16);
    pointerKind = cudaMemoryTypeHost;
    for (int band = 0; band < 4; ++band) {
        failLaunch = band;
        check(render(ARTF_CUDA_EXACT, buffer, 16, 16, 64) == ARTF_CUDA_ELAUNCH, "a failed launch is reported");
        check(launches == band + 1 && pendingLaunches == 0, "the bands before it went out, and none is in flight");
        check(strstr(artfCudaLastError(), "trace launch") != nullptr, "the launch's error is the one reported");
    }
    failLaunch = -1;
    failEvent = 1;
    check(render(ARTF_CUDA_EXACT, buffer, 16, 16, 0) == ARTF_CUDA_ELAUNCH && launches == 1, "a failed event is reported");
    check(pendingLaunches == 0, "a failed call left a kernel in flight that writes the caller's buffer");
    check(strstr(artfCudaLastError(), "cudaEventRecord") != nullptr, "the event's error is the one reported");
    failEvent = -1;
    free(buffer);
}

/* Gases' memory: plain device memory, kept for the context's next gases up to two, its own context's alone, and
 * all given back whichever goes first. */
static void gasMemory() {
    ArtfCuda *a = nullptr, *b = nullptr;
    check(artfCudaCreate(0, &a) == ARTF_CUDA_OK && artfCudaCreate(0, &b) == ARTF_CUDA_OK, "two contexts");
    const size_t before = live.size();
    void *block[4], *again, *other, *late;
    artf::GasStore *store[4], *s, *so, *sl;
    for (int k = 0; k < 4; ++k)
        check(artf::takeGas(a, 1024, &block[k], &store[k]) == cudaSuccess && live.count(block[k]), "a gas's memory");
    for (int k = 0; k < 4; ++k) artf::giveGas(store[k], block[k], true);
    check(live.size() == before + 2, "two gases' memory kept");
    check(artf::takeGas(b, 1024, &other, &so) == cudaSuccess && live.size() == before + 3, "another context's is its own");
    check(artf::takeGas(a, 1024, &again, &s) == cudaSuccess && live.size() == before + 3, "kept memory taken again");
    check(artf::takeGas(a, 1024, &late, &sl) == cudaSuccess && late != again && live.size() == before + 3, "and the other");
    artf::giveGas(s, again, false);
    check(live.count(again) == 0 && live.size() == before + 2, "memory that may be in use is not kept");
    artfCudaDestroy(a);
    check(live.count(late) == 1, "a context gives back what it keeps, not what a gas holds");
    artf::giveGas(sl, late, true); /* (its context is gone) */
    check(live.count(late) == 0, "a gas that outlived its context gives its memory back");
    artf::giveGas(so, other, true);
    artfCudaDestroy(b);
    check(live.count(other) == 0, "nothing left");
    failMalloc = true;
    check(artf::takeGas(ctx, 1024, &late, &sl) == cudaErrorMemoryAllocation && !late, "a failed allocation is reported");
    failMalloc = false;
}

int main() {
    inputs = (float*)calloc(ARTF_CUDA_MAP_FLOATS, sizeof(float));
    check(artfCudaCreate(0, &ctx) == ARTF_CUDA_OK, "a context");
    hostFrames();
    failedCalls();
    gasMemory();
    artfCudaDestroy(ctx);
    check(live.empty(), "device memory left after the context");
    free(inputs);
    printf("host checks failed: %d\n", failures);
    return failures != 0;
}
