/* A stand-in for the CUDA runtime, preloaded into a process that has no GPU
 * (tests/test_host_paths_cpu.py): device memory is host memory with a limit,
 * kernels do nothing, and the fake_* calls make single calls fail and say what
 * happened.  It covers what liblbm_gb300.so calls. */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>

static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;
static __thread cudaError_t last_error;
static __thread enum cudaStreamCaptureMode thread_mode = cudaStreamCaptureModeGlobal;
static cudaError_t err(cudaError_t e)
{
    if (e != cudaSuccess) last_error = e;
    return e;
}

/* ---- memory ---- */
static struct { char* p; size_t bytes; } blocks[4096];
static int nblocks;
static size_t total = (size_t)280 << 30, used;
static int capture_elsewhere, capture_broken;

void fake_memory(size_t bytes) { total = bytes; }
size_t fake_used(void) { return used; }
/* Another thread's stream is being captured in global mode: calls that such a capture forbids break it. */
void fake_capture_elsewhere(int on) { capture_elsewhere = on, capture_broken = 0; }
int fake_capture_broken(void) { return capture_broken; }
/* 1 if the address lies in live device memory. */
int fake_live(const void* at)
{
    int found = 0;
    pthread_mutex_lock(&mu);
    for (int i = 0; i < nblocks; ++i)
        if ((const char*)at >= blocks[i].p && (const char*)at < blocks[i].p + blocks[i].bytes) found = 1;
    pthread_mutex_unlock(&mu);
    return found;
}
static int forbidden(void)
{
    if (!capture_elsewhere || thread_mode == cudaStreamCaptureModeRelaxed) return 0;
    capture_broken = 1;
    return 1;
}
cudaError_t cudaMalloc(void** p, size_t bytes)
{
    cudaError_t e = cudaSuccess;
    if (forbidden()) return err(cudaErrorStreamCaptureUnsupported);
    pthread_mutex_lock(&mu);
    if (used + bytes > total || nblocks == 4096) e = cudaErrorMemoryAllocation;
    else {
        char* q = mmap(NULL, bytes ? bytes : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
        if (q == MAP_FAILED) e = cudaErrorMemoryAllocation;
        else {
            blocks[nblocks].p = q;
            blocks[nblocks++].bytes = bytes ? bytes : 1;
            used += bytes;
            *p = q;
        }
    }
    pthread_mutex_unlock(&mu);
    return err(e);
}
cudaError_t cudaFree(void* p)
{
    if (!p) return cudaSuccess;
    if (forbidden()) return err(cudaErrorStreamCaptureUnsupported);
    pthread_mutex_lock(&mu);
    int i = 0;
    while (i < nblocks && blocks[i].p != p) ++i;
    if (i == nblocks) {
        fprintf(stderr, "cudaFree of an unknown pointer\n");
        abort();
    }
    munmap(p, blocks[i].bytes);
    used -= blocks[i].bytes;
    blocks[i] = blocks[--nblocks];
    pthread_mutex_unlock(&mu);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t)
{
    *f = total > used ? total - used : 0;
    *t = total;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned flags) { return (*p = calloc(1, bytes)) ? cudaSuccess : err(cudaErrorMemoryAllocation); }
cudaError_t cudaMallocHost(void** p, size_t bytes) { return cudaHostAlloc(p, bytes, 0); }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned flags) { *d = h; return cudaSuccess; }

/* ---- copies ---- */
static int fail_copies;
void fake_fail_copies(int n) { fail_copies = n; } /* the next n copies to the host */
static cudaError_t copied(void* d, const void* s, size_t n, enum cudaMemcpyKind k)
{
    if (k == cudaMemcpyDeviceToHost && fail_copies > 0) return --fail_copies, err(cudaErrorInvalidValue);
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) { return copied(d, s, n, k); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
    return k == cudaMemcpyDeviceToDevice ? cudaSuccess : copied(d, s, n, k);
}
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) { return cudaMemset(d, v, n); }
cudaError_t cudaMemcpy3D(const struct cudaMemcpy3DParms* p)
{
    if (p->kind == cudaMemcpyDeviceToHost && fail_copies > 0) return --fail_copies, err(cudaErrorInvalidValue);
    for (size_t z = 0; z < p->extent.depth; ++z)
        for (size_t y = 0; y < p->extent.height; ++y)
            memcpy((char*)p->dstPtr.ptr + ((p->dstPos.z + z) * p->dstPtr.ysize + p->dstPos.y + y) * p->dstPtr.pitch + p->dstPos.x,
                   (char*)p->srcPtr.ptr + ((p->srcPos.z + z) * p->srcPtr.ysize + p->srcPos.y + y) * p->srcPtr.pitch + p->srcPos.x,
                   p->extent.width);
    return cudaSuccess;
}
cudaError_t cudaMemcpy3DAsync(const struct cudaMemcpy3DParms* p, cudaStream_t st) { return cudaMemcpy3D(p); }

/* ---- kernels ---- */
typedef void (*launch_fn)(const char* name, void** args);
static struct { const void* fn; const char* name; } kernels[2048];
static int nkernels;
static launch_fn on_launch;
static const char* fail_name;
static int fail_at;
void fake_on_launch(launch_fn f) { on_launch = f; }
/* The at-th launch (from 1) of a kernel whose mangled name contains `name` fails. */
void fake_fail_launch(const char* name, int at) { fail_name = name ? strdup(name) : NULL, fail_at = at; }
static cudaError_t launched(const void* fn, void** args)
{
    const char* name = "?";
    for (int i = 0; i < nkernels; ++i)
        if (kernels[i].fn == fn) name = kernels[i].name;
    if (fail_name && strstr(name, fail_name) && --fail_at == 0) return err(cudaErrorLaunchOutOfResources);
    if (strstr(name, "bounded_wait_probe")) **(int**)args[0] |= 1;              /* (err, limit) */
    if (strstr(name, "compute_macros")) **(int**)args[7] = **(int**)args[6];    /* (..., err, host_err) */
    if (on_launch) on_launch(name, args);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void** args) { return launched(fn, args); }
cudaError_t __cudaLaunchKernel(const void* fn, dim3 g, dim3 b, void** args, size_t s, cudaStream_t st) { return launched(fn, args); }
cudaError_t __cudaGetKernel(const void** k, const void* fn) { *k = fn; return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st)
{
    g->x = g->y = g->z = b->x = b->y = b->z = 1;
    *s = 0;
    *(void**)st = NULL;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void* f) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) {}
void __cudaUnregisterFatBinary(void** h) {}
void __cudaRegisterFunction(void** h, const char* fn, char* dev, const char* name, int n, void* a, void* b, void* c, void* d, int* e)
{
    if (nkernels < 2048) kernels[nkernels].fn = fn, kernels[nkernels++].name = name;
}
void __cudaRegisterVar(void** h, char* v, char* dev, const char* name, int a, size_t b, int c, int d) {}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* fn) { memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* fn, enum cudaFuncAttribute a, int v) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* fn, int b, size_t s, unsigned f) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* sym) { return err(cudaErrorInvalidSymbol); }

/* ---- device ---- */
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return forbidden() ? err(cudaErrorStreamCaptureUnsupported) : cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 232448;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = last_error;
    last_error = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return "fake error"; }
static int encode() { return 0; }
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** p, unsigned v, unsigned long long f,
                                             enum cudaDriverEntryPointQueryResult* q)
{
    *p = strcmp(name, "cuTensorMapEncodeTiled") ? NULL : (void*)encode;
    if (q) *q = *p ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}

/* ---- streams, events, graphs ---- */
static cudaStream_t capturing = (cudaStream_t)-1;
void fake_capturing(cudaStream_t st) { capturing = st; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) { *s = malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus* c)
{
    *c = s == capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(enum cudaStreamCaptureMode* m)
{
    const enum cudaStreamCaptureMode was = thread_mode;
    thread_mode = *m;
    *m = was;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) { *g = malloc(1); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long f) { *x = malloc(1); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { free(x); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) { *ms = 1; return cudaSuccess; }
