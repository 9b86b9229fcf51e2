/* A CUDA runtime without a GPU, preloaded over the real one by
 * tests/test_host_failures_cpu.py: device memory is host memory, a launch is
 * noted by the kernel's name and runs nothing, and the calls that a test names
 * fail.  It lets the library's host code meet errors that no GPU should be
 * driven to. */
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define MAX_BLOCKS 4096
#define MAX_KERNELS 1024

static struct { void* p; size_t n; } blocks[MAX_BLOCKS];
static struct { const void* f; char name[256]; } kernels[MAX_KERNELS];
static int kernel_count;
static char launches[1 << 20];
static size_t launches_len;
static cudaError_t last = cudaSuccess;

/* ---- what a test sets and reads ---- */
size_t fake_memory = (size_t)-1;   /* bytes of device memory */
int fake_sync_error = 0;           /* the next synchronisations fail with it */
int fake_copy_error = 0;           /* the next copies to the host */
int fake_capturing = 0;            /* streams are being captured */
int fake_clusters = 1;             /* clusters that can be resident */

size_t fake_used(void) {
    size_t used = 0;
    for (int i = 0; i < MAX_BLOCKS; ++i) used += blocks[i].p ? blocks[i].n : 0;
    return used;
}
/* size of the live block at p, 0 for any other address */
size_t fake_block(const void* p) {
    for (int i = 0; i < MAX_BLOCKS; ++i)
        if (p && blocks[i].p == p) return blocks[i].n;
    return 0;
}
/* the launched kernels' mangled names, a line each; clears them */
const char* fake_launches(void) {
    static char out[sizeof launches];
    memcpy(out, launches, launches_len);
    out[launches_len] = 0;
    launches_len = 0;
    return out;
}

static cudaError_t result(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
static cudaError_t launched(const void* f) {
    for (int i = 0; i < kernel_count; ++i)
        if (kernels[i].f == f) {
            const size_t n = strlen(kernels[i].name);
            if (launches_len + n + 2 < sizeof launches) {
                memcpy(launches + launches_len, kernels[i].name, n);
                launches[launches_len + n] = '\n';
                launches_len += n + 1;
            }
            return cudaSuccess;
        }
    return result(cudaErrorInvalidDeviceFunction);
}

/* ---- registration and launches ---- */
void** __cudaRegisterFatBinary(void* fat) { static void* h; (void)fat; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterVar(void** h, char* hv, char* da, const char* dn, int ext, size_t n, int c, int g) {
    (void)h; (void)hv; (void)da; (void)dn; (void)ext; (void)n; (void)c; (void)g;
}
void __cudaRegisterFunction(void** h, const char* f, char* df, const char* name, int limit, void* tid,
                            void* bid, void* bd, void* gd, int* ws) {
    (void)h; (void)df; (void)limit; (void)tid; (void)bid; (void)bd; (void)gd; (void)ws;
    if (kernel_count == MAX_KERNELS) abort();
    kernels[kernel_count].f = f;
    snprintf(kernels[kernel_count++].name, sizeof kernels[0].name, "%s", name);
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) {
    (void)g; (void)b; (void)s; (void)st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
    const dim3 one = {1, 1, 1};
    *g = *b = one;
    *s = 0;
    *(void**)st = NULL;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void** a, size_t s, cudaStream_t st) {
    (void)g; (void)b; (void)a; (void)s; (void)st;
    return launched((const void*)k);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
    (void)a;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension && fake_clusters == 0)
            return result(cudaErrorLaunchOutOfResources);
    return launched(f);
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
    (void)f; (void)a; (void)v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t s,
                                                                   unsigned fl) {
    (void)f; (void)b; (void)s; (void)fl;
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
    (void)f; (void)c;
    *n = fake_clusters;
    return cudaSuccess;
}

/* ---- memory ---- */
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = NULL;
    if (n == 0) return cudaSuccess;
    if (fake_capturing) return result(cudaErrorStreamCaptureUnsupported);
    if (n > fake_memory || fake_used() > fake_memory - n) return result(cudaErrorMemoryAllocation);
    for (int i = 0; i < MAX_BLOCKS; ++i)
        if (blocks[i].p == NULL) {
            if ((blocks[i].p = calloc(1, n)) == NULL) return result(cudaErrorMemoryAllocation);
            blocks[i].n = n;
            *p = blocks[i].p;
            return cudaSuccess;
        }
    return result(cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void* p) {
    if (p == NULL) return cudaSuccess;
    for (int i = 0; i < MAX_BLOCKS; ++i)
        if (blocks[i].p == p) {
            free(p);
            blocks[i].p = NULL;
            return cudaSuccess;
        }
    return result(cudaErrorInvalidValue);
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned f) {
    (void)f;
    *p = calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) {
    if (k == cudaMemcpyDeviceToHost && fake_copy_error) return result((cudaError_t)fake_copy_error);
    if (n) memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
    (void)st;
    return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    if (n) memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    (void)st;
    return cudaMemset(d, v, n);
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { (void)s; *p = NULL; return cudaErrorInvalidSymbol; }

/* ---- device, streams, events, graphs ---- */
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp* p, int d) {
    (void)d;
    memset(p, 0, sizeof *p);
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorName(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
const char* cudaGetErrorString(cudaError_t e) { return cudaGetErrorName(e); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
    (void)f;
    *s = (cudaStream_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    (void)s;
    return fake_sync_error ? result((cudaError_t)fake_sync_error) : cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus* st) {
    (void)s;
    *st = fake_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) {
    (void)s; (void)m;
    fake_capturing = 1;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    (void)s;
    fake_capturing = 0;
    *g = (cudaGraph_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long f) {
    (void)g; (void)f;
    *x = (cudaGraphExec_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) { (void)x; (void)s; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { free(x); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
    (void)a; (void)b;
    *ms = 1.f;
    return cudaSuccess;
}
