/* A CUDA runtime without a device, for CPU tests of the library's host code:
 * the library's objects are linked with this file in place of cudart.  Memory is
 * host memory, launches only record the kernel's name, and a test may have
 * allocations or cooperative launches fail.  Blocks from BIG bytes on are
 * address space that nothing touches: copies and fills of that size are left
 * out. */
#define _GNU_SOURCE
#include <driver_types.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>
#include <vector_types.h>

#define BIG ((size_t)64 << 20)
#define API __attribute__((visibility("default")))

/* ---- the test's side ---- */
static long g_mallocs, g_fail_from = -1;
static int g_coop_error;
static char g_log[1 << 20];
static size_t g_log_len;

API long fake_mallocs(void) { return g_mallocs; }
/* every allocation from the n-th on (counted from 0 at this call) fails; < 0: none */
API void fake_fail_mallocs_from(long n) { g_mallocs = 0; g_fail_from = n; }
API void fake_coop_error(int e) { g_coop_error = e; }
API void fake_log_clear(void) { g_log_len = 0; g_log[0] = 0; }
API const char *fake_log(void) { return g_log; }

/* ---- kernels ---- */
typedef struct { const void *fn; const char *name; size_t smem; int carveout; } Kernel;
static Kernel g_kernels[4096];
static int g_nkernels;

/* of the kernel whose name contains `name`: dynamic shared memory of its last
 * launch, and its preferred carve-out in percent (0: never set) */
static Kernel *by_name(const char *name)
{
    for (int i = 0; i < g_nkernels; i++)
        if (strstr(g_kernels[i].name, name)) return &g_kernels[i];
    abort();
}
API long fake_smem(const char *name) { return (long)by_name(name)->smem; }
API int fake_carveout(const char *name) { return by_name(name)->carveout; }
static size_t g_shared_size;
/* static shared memory of every kernel */
API void fake_shared_size(long n) { g_shared_size = (size_t)n; }

static void log_line(const char *s)
{
    const size_t n = strlen(s);
    if (g_log_len + n + 2 > sizeof(g_log)) abort();
    memcpy(g_log + g_log_len, s, n);
    g_log_len += n;
    g_log[g_log_len++] = '\n';
    g_log[g_log_len] = 0;
}

static cudaError_t launched(const void *fn, size_t smem)
{
    for (int i = 0; i < g_nkernels; i++)
        if (g_kernels[i].fn == fn)
        {
            g_kernels[i].smem = smem;
            log_line(g_kernels[i].name);
            return cudaSuccess;
        }
    return cudaErrorInvalidDeviceFunction;
}

API void **__cudaRegisterFatBinary(void *b) { static void *h; (void)b; return &h; }
API void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
API void __cudaUnregisterFatBinary(void **h) { (void)h; }
API void __cudaRegisterVar(void **h, char *v, char *a, const char *n, int e, size_t s, int c, int g)
{
    (void)h; (void)v; (void)a; (void)n; (void)e; (void)s; (void)c; (void)g;
}
API void __cudaRegisterFunction(void **h, const char *fn, char *dev, const char *name, int lim, uint3 *t, uint3 *b,
                                dim3 *bd, dim3 *gd, int *ws)
{
    (void)h; (void)dev; (void)lim; (void)t; (void)b; (void)bd; (void)gd; (void)ws;
    if (g_nkernels == 4096) abort();
    g_kernels[g_nkernels].fn = fn;
    g_kernels[g_nkernels++].name = name;
}
static dim3 g_grid, g_block;
static size_t g_smem;
static void *g_stream;
API unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void *s)
{
    g_grid = g; g_block = b; g_smem = smem; g_stream = s;
    return 0;
}
API cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s)
{
    *g = g_grid; *b = g_block; *smem = g_smem; *(void **)s = g_stream;
    return cudaSuccess;
}
API cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fn) { *k = (cudaKernel_t)fn; return cudaSuccess; }
API cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **a, size_t m, cudaStream_t s)
{
    (void)g; (void)b; (void)a; (void)s;
    return launched((const void *)k, m);
}
API cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **a, size_t m, cudaStream_t s)
{
    (void)g; (void)b; (void)a; (void)s;
    return launched(f, m);
}
API cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a)
{
    (void)a;
    return launched(f, c->dynamicSmemBytes);
}
API cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **a, size_t m, cudaStream_t s)
{
    (void)g; (void)b; (void)a; (void)s;
    return g_coop_error ? (cudaError_t)g_coop_error : launched(f, m);
}
API cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v)
{
    for (int i = 0; i < g_nkernels; i++)
        if (g_kernels[i].fn == f && a == cudaFuncAttributePreferredSharedMemoryCarveout) g_kernels[i].carveout = v;
    return cudaSuccess;
}
API cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes *a, const void *f)
{
    (void)f;
    memset(a, 0, sizeof(*a));
    a->sharedSizeBytes = g_shared_size;
    return cudaSuccess;
}
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int t, size_t m)
{
    (void)f; (void)t; (void)m;
    *n = 2;
    return cudaSuccess;
}

/* ---- memory ---- */
API cudaError_t cudaMalloc(void **p, size_t n)
{
    *p = NULL;
    if (g_fail_from >= 0 && g_mallocs >= g_fail_from) return cudaErrorMemoryAllocation;
    g_mallocs++;
    /* never given back: blocks keep distinct addresses */
    *p = mmap(NULL, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    return *p == MAP_FAILED ? (*p = NULL, cudaErrorMemoryAllocation) : cudaSuccess;
}
API cudaError_t cudaFree(void *p) { (void)p; return cudaSuccess; }
API cudaError_t cudaHostAlloc(void **p, size_t n, unsigned f) { (void)f; *p = calloc(1, n); return cudaSuccess; }
API cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
API cudaError_t cudaHostRegister(void *p, size_t n, unsigned f) { (void)p; (void)n; (void)f; return cudaSuccess; }
API cudaError_t cudaHostUnregister(void *p) { (void)p; return cudaSuccess; }
API cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k)
{
    (void)k;
    if (n < BIG) memcpy(d, s, n);
    return cudaSuccess;
}
API cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
    (void)st;
    return cudaMemcpy(d, s, n, k);
}
API cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h,
                                  enum cudaMemcpyKind k, cudaStream_t st)
{
    (void)k; (void)st;
    for (size_t i = 0; i < h; i++) memcpy((char *)d + i * dp, (const char *)s + i * sp, w);
    return cudaSuccess;
}
API cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t s)
{
    (void)s;
    if (n < BIG) memset(d, v, n);
    return cudaSuccess;
}
API cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p)
{
    (void)p;
    memset(a, 0, sizeof(*a));
    return cudaSuccess;
}
API cudaError_t cudaGetSymbolAddress(void **p, const void *s)
{
    (void)s;
    *p = NULL;
    return cudaErrorInvalidSymbol;
}

/* ---- device, streams, events, graphs ---- */
API cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
API cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
API cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
API cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d)
{
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 233472 : 0;
    return cudaSuccess;
}
API cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
API cudaError_t cudaGetLastError(void) { return cudaSuccess; }
API const char *cudaGetErrorString(cudaError_t e) { (void)e; return "an error the test asked for"; }
API cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)calloc(1, 8); return cudaSuccess; }
API cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
API cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
API cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return cudaSuccess; }
API cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; *g = (cudaGraph_t)calloc(1, 8); return cudaSuccess; }
API cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)calloc(1, 8); return cudaSuccess; }
API cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; return cudaEventCreate(e); }
API cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
API cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
API cudaError_t cudaEventQuery(cudaEvent_t e) { (void)e; return cudaSuccess; }
API cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *ms = 0.1f; return cudaSuccess; }
API cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long f) { (void)g; (void)f; log_line("<instantiate>"); *x = (cudaGraphExec_t)calloc(1, 8); return cudaSuccess; }
API cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
API cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { free(x); return cudaSuccess; }
API cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) { (void)x; (void)s; log_line("<graph>"); return cudaSuccess; }
