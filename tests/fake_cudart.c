/* A CUDA runtime without a GPU, for tests of the host code (LD_PRELOAD).
 *
 * Device memory is host memory within a limit that the test sets, copies and
 * fills are done at once, streams and events do nothing, and a kernel launch is
 * only recorded: its name, grid, block and dynamic shared memory.  Limits and
 * occupancy are a B200's, with 128 registers a thread and FAKE_STATIC bytes of
 * static shared memory a CTA.
 */
#define _GNU_SOURCE
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <cuda_runtime_api.h>

#define FAKE_SMS 148
#define FAKE_OPTIN 232448
#define FAKE_SM_SMEM 233472
#define FAKE_STATIC 1008

/* ---- kernels by name, launches ------------------------------------------ */
static struct { const void* fn; char name[512]; } kernels[1024];
static int n_kernels;
static struct { const char* name; int grid, block; size_t smem; } launches[4096];
static int n_launches;

void** __cudaRegisterFatBinary(void* p) { (void)p; static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterVar(void** h, char* v, char* a, const char* n, int e, size_t s, int c, int g) {
    (void)h; (void)v; (void)a; (void)n; (void)e; (void)s; (void)c; (void)g;
}
void __cudaRegisterFunction(void** h, const char* fn, char* dfn, const char* name, int tl, uint3* tid, uint3* bid,
                            dim3* bd, dim3* gd, int* ws) {
    (void)h; (void)dfn; (void)tl; (void)tid; (void)bid; (void)bd; (void)gd; (void)ws;
    if (n_kernels < 1024) {
        kernels[n_kernels].fn = fn;
        snprintf(kernels[n_kernels++].name, sizeof(kernels[0].name), "%s", name);
    }
}
static const char* name_of(const void* fn) {
    for (int i = 0; i < n_kernels; ++i)
        if (kernels[i].fn == fn) return kernels[i].name;
    return "?";
}
static cudaError_t record(const void* fn, dim3 grid, dim3 block, size_t smem) {
    if (n_launches < 4096) {
        launches[n_launches].name = name_of(fn);
        launches[n_launches].grid = (int)grid.x;
        launches[n_launches].block = (int)block.x;
        launches[n_launches++].smem = smem;
    }
    return cudaSuccess;
}
int fake_launches(void) { return n_launches; }
void fake_clear_launches(void) { n_launches = 0; }
const char* fake_launch(int i, int* grid, int* block, size_t* smem) {
    *grid = launches[i].grid;
    *block = launches[i].block;
    *smem = launches[i].smem;
    return launches[i].name;
}

static struct { dim3 g, b; size_t m; cudaStream_t s; } conf;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s) {
    conf.g = g; conf.b = b; conf.m = m; conf.s = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
    *g = conf.g; *b = conf.b; *m = conf.m; *(cudaStream_t*)s = conf.s;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 g, dim3 b, void** args, size_t m, cudaStream_t s) {
    (void)args; (void)s;
    return record(fn, g, b, m);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void** args) {
    (void)args;
    return record(fn, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}

/* ---- memory ---------------------------------------------------------------- */
static size_t mem_limit = (size_t)8 << 30, mem_used;
struct head { size_t bytes; size_t pad; };
void fake_set_memory(size_t bytes) { mem_limit = bytes; }
size_t fake_memory_used(void) { return mem_used; }
cudaError_t cudaMalloc(void** p, size_t bytes) {
    if (mem_used + bytes > mem_limit) return cudaErrorMemoryAllocation;
    struct head* h = malloc(sizeof(struct head) + bytes);
    if (!h) return cudaErrorMemoryAllocation;
    h->bytes = bytes;
    mem_used += bytes;
    *p = h + 1;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (p) {
        struct head* h = (struct head*)p - 1;
        mem_used -= h->bytes;
        free(h);
    }
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    *f = mem_limit - mem_used;
    *t = mem_limit;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned fl) { (void)fl; *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned fl) { (void)fl; *d = h; return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) { (void)k; memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
    (void)k; (void)st;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) { (void)st; memset(d, v, n); return cudaSuccess; }

/* ---- device, kernels' limits ----------------------------------------------- */
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount ? FAKE_SMS : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? FAKE_OPTIN : 0;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
    (void)f;
    return a == cudaFuncAttributeMaxDynamicSharedMemorySize && v + FAKE_STATIC > FAKE_OPTIN ? cudaErrorInvalidValue
                                                                                            : cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* f) {
    (void)f;
    memset(a, 0, sizeof(*a));
    a->sharedSizeBytes = FAKE_STATIC;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int threads, size_t smem) {
    (void)f;
    const int by_regs = 65536 / (128 * threads), by_smem = (int)(FAKE_SM_SMEM / (smem + FAKE_STATIC + 1024));
    *n = by_regs < by_smem ? by_regs : by_smem;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int threads, size_t smem,
                                                                   unsigned fl) {
    (void)fl;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, f, threads, smem);
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, (int)c->blockDim.x, c->dynamicSmemBytes);
    *n = per * FAKE_SMS / (int)c->attrs[0].val.clusterDim.x;
    return cudaSuccess;
}

/* ---- streams, events ------------------------------------------------------- */
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned fl) { (void)fl; *s = (cudaStream_t)(uintptr_t)16; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned fl) { (void)s; (void)e; (void)fl; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)(uintptr_t)16; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned fl) { (void)fl; return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *ms = 1.0f; return cudaSuccess; }
