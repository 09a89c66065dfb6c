/* A stand-in for the CUDA runtime: the library's objects linked against this file run their host code on a
 * machine without a GPU.  "Device" memory is host memory, copies are memcpy, kernels are recorded and not
 * run, and an allocation can be told to fail.  tests/fake_cuda.py builds and drives it. */
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define MAX_KERNELS 4096
#define MAX_LAUNCHES 65536

static struct { const void *host; const char *name; } kernels[MAX_KERNELS];
static int nkernels;
static struct { const char *name; unsigned grid, block; } launches[MAX_LAUNCHES];
static int nlaunches, live, fail_in = -1;

int fake_launches(void) { return nlaunches; }
const char *fake_launch_name(int i) { return launches[i].name; }
unsigned fake_launch_grid(int i) { return launches[i].grid; }
void fake_reset(void) { nlaunches = 0; }
/* The n-th device allocation from now on fails (0: the next one; negative: none). */
void fake_fail_malloc(int n) { fail_in = n; }
int fake_live_allocations(void) { return live; }

/* The library's operator new: the largest request since fake_largest_new() was last read. */
static size_t largest_new;
size_t fake_largest_new(void) { const size_t n = largest_new; largest_new = 0; return n; }
void *_Znwm(size_t n) { if (n > largest_new) largest_new = n; void *p = malloc(n ? n : 1); if (!p) abort(); return p; }
void _ZdlPv(void *p) { free(p); }
void _ZdlPvm(void *p, size_t n) { (void)n; free(p); }

static void record(const void *f, dim3 grid, dim3 block) {
    const char *name = "?";
    for (int i = 0; i < nkernels; ++i)
        if (kernels[i].host == f) name = kernels[i].name;
    if (nlaunches < MAX_LAUNCHES) {
        launches[nlaunches].name = name;
        launches[nlaunches].grid = grid.x * grid.y * grid.z;
        launches[nlaunches++].block = block.x * block.y * block.z;
    }
}

/* ---- what nvcc's host stubs call ---- */
struct symbol { const void *host; size_t size; void *mem; };
static struct symbol symbols[64];
static int nsymbols;
static struct { dim3 grid, block; size_t smem; void *stream; } pending;

void **__cudaRegisterFatBinary(void *bin) { (void)bin; static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void **h, const char *host, char *dev, const char *name, int limit, void *tid, void *bid,
                            void *bdim, void *gdim, int *wsize) {
    (void)h; (void)dev; (void)limit; (void)tid; (void)bid; (void)bdim; (void)gdim; (void)wsize;
    if (nkernels < MAX_KERNELS) {
        kernels[nkernels].host = host;
        kernels[nkernels++].name = name;
    }
}
void __cudaRegisterVar(void **h, char *host, char *dev, const char *name, int ext, size_t size, int constant, int global) {
    (void)h; (void)dev; (void)name; (void)ext; (void)constant; (void)global;
    if (nsymbols < 64) {
        symbols[nsymbols].host = host;
        symbols[nsymbols++].size = size;
    }
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void *stream) {
    pending.grid = grid; pending.block = block; pending.smem = smem; pending.stream = stream;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = pending.grid; *block = pending.block; *smem = pending.smem; *(void **)stream = pending.stream;
    return cudaSuccess;
}

size_t fake_symbol_bytes(void) {
    size_t n = 0;
    for (int i = 0; i < nsymbols; ++i) n += symbols[i].size;
    return n;
}

/* ---- runtime ---- */
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t st) {
    (void)args; (void)smem; (void)st;
    record(f, grid, block);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
    (void)args;
    record(f, c->gridDim, c->blockDim);
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
    *p = NULL;
    if (fail_in >= 0 && fail_in-- == 0) return cudaErrorMemoryAllocation;
    if (posix_memalign(p, 256, n ? n : 1)) return cudaErrorMemoryAllocation;
    ++live;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) { if (p) --live; free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned flags) { (void)flags; return posix_memalign(p, 256, n ? n : 1) ? cudaErrorMemoryAllocation : cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
/* Work of the default stream that other streams do not wait for: copies from pageable memory, memsets. */
static int unfinished;
int fake_unfinished(void) { return unfinished; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) { memcpy(d, s, n); unfinished += k == cudaMemcpyHostToDevice; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) { (void)k; (void)st; memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { memset(d, v, n); ++unfinished; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) { (void)st; memset(d, v, n); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *sym) {
    for (int i = 0; i < nsymbols; ++i)
        if (symbols[i].host == sym) {
            if (!symbols[i].mem) symbols[i].mem = calloc(1, symbols[i].size);
            *p = symbols[i].mem;
            return cudaSuccess;
        }
    return cudaErrorInvalidSymbol;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { static char s[32]; snprintf(s, sizeof s, "fake error %d", (int)e); return s; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return d == 0 ? cudaSuccess : cudaErrorInvalidDevice; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(struct cudaDeviceProp *p, int d) {
    (void)d;
    memset(p, 0, sizeof *p);
    p->multiProcessorCount = 148;
    p->major = 10;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { unfinished = 0; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { if (!s) unfinished = 0; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) { (void)f; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int t, size_t smem) {
    (void)f; (void)t; (void)smem;
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p) {
    memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeDevice;
    a->devicePointer = (void *)p;
    return cudaSuccess;
}
cudaError_t cudaLaunchHostFunc(cudaStream_t s, cudaHostFn_t f, void *u) { (void)s; f(u); return cudaSuccess; }
static int encode_ok(void) { return 0; }
cudaError_t cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long flags, enum cudaDriverEntryPointQueryResult *r) {
    (void)name; (void)flags;
    *f = (void *)encode_ok;
    if (r) *r = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
