/* A stand-in for the CUDA runtime, preloaded in front of the real one by tests of the library's host
 * code (test_host_runtime.py): FAKE_DEVICES devices whose memory is host memory, kernels that do
 * nothing, and the checks of the real runtime that depend on the calling thread's device: a launch
 * goes to a stream of the current device, and needs the opt-in of that device for more than 48 KB of
 * dynamic shared memory.  Grids are checked too: at most 65535 blocks along y and z.  fake_fail() makes a later call fail; fake_live() counts what is allocated. */
#define _GNU_SOURCE
#include <stddef.h>
#include <stdlib.h>
#include <string.h>
#include <cuda_runtime_api.h>
/* the launch entry points that nvcc's host code calls */
typedef struct {
    unsigned x, y, z;
} Dim;

enum { MAXDEV = 4, MAXFUNC = 4096, MAXBUF = 1 << 16 };
struct stream {
    int dev;
};
static __thread int cur;
static int ndev;
static struct {
    char *p;
    size_t n;
    int dev;
} bufs[MAXBUF];
static struct {
    const void *f;
    int bytes[MAXDEV];
} funcs[MAXFUNC];
static int nfuncs;
static long long launches, fail_at[2] = {-1, -1}; /* mallocs, launches */
static cudaError_t last;

static cudaError_t ret(cudaError_t e)
{
    if (e != cudaSuccess) last = e;
    return e;
}
static int fails(int kind) { return fail_at[kind] >= 0 && fail_at[kind]-- == 0; }

/* for the tests: the n-th malloc (kind 0) or launch (kind 1) from now fails; n < 0: none */
void fake_fail(int kind, long long n) { fail_at[kind] = n; }
long long fake_launches(void) { return launches; }
long long fake_live(int dev)
{
    long long s = 0;
    for (int i = 0; i < MAXBUF; ++i)
        if (bufs[i].p && bufs[i].dev == dev) s += (long long)bufs[i].n;
    return s;
}

cudaError_t cudaGetDeviceCount(int *n)
{
    const char *e = getenv("FAKE_DEVICES");
    ndev = e ? atoi(e) : 1;
    *n = ndev;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d)
{
    int n;
    cudaGetDeviceCount(&n);
    if (d < 0 || d >= n) return ret(cudaErrorInvalidDevice);
    cur = d;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d)
{
    *d = cur;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int dev)
{
    (void)dev;
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrL2CacheSize ? 129 << 20 : 1;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp *p, int dev)
{
    (void)dev;
    memset(p, 0, sizeof *p);
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "fake error"; }
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}

cudaError_t cudaMalloc(void **p, size_t n)
{
    *p = NULL;
    if (fails(0)) return ret(cudaErrorMemoryAllocation);
    for (int i = 0; i < MAXBUF; ++i)
        if (!bufs[i].p) {
            bufs[i].p = calloc(1, n ? n : 1);
            if (!bufs[i].p) break;
            bufs[i].n = n;
            bufs[i].dev = cur;
            *p = bufs[i].p;
            return cudaSuccess;
        }
    return ret(cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void *p)
{
    if (!p) return cudaSuccess;
    for (int i = 0; i < MAXBUF; ++i)
        if (bufs[i].p == p) {
            free(p);
            bufs[i].p = NULL;
            return cudaSuccess;
        }
    return ret(cudaErrorInvalidValue);
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t)
{
    *f = *t = (size_t)1 << 38;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k)
{
    (void)k;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
    (void)st;
    return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st)
{
    (void)st;
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbolAsync(const void *y, const void *s, size_t n, size_t o, enum cudaMemcpyKind k, cudaStream_t st)
{
    (void)y, (void)s, (void)n, (void)o, (void)k, (void)st;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *y)
{
    *p = (void *)y;
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f)
{
    struct stream *q = malloc(sizeof *q);
    (void)f;
    q->dev = cur;
    *s = (cudaStream_t)q;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s, (void)e, (void)f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s, (void)m; return ret(cudaErrorNotSupported); }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; *g = NULL; return ret(cudaErrorNotSupported); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long f) { (void)x, (void)g, (void)f; return ret(cudaErrorNotSupported); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) { (void)x, (void)s; return ret(cudaErrorNotSupported); }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { (void)x; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f)
{
    (void)f;
    *e = (cudaEvent_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e, (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b)
{
    (void)a, (void)b;
    *ms = 1.0f;
    return cudaSuccess;
}

static int func_at(const void *f)
{
    for (int i = 0; i < nfuncs; ++i)
        if (funcs[i].f == f) return i;
    if (nfuncs == MAXFUNC) abort();
    funcs[nfuncs].f = f;
    return nfuncs++;
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v)
{
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) funcs[func_at(f)].bytes[cur] = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t s, unsigned fl)
{
    (void)f, (void)b, (void)s, (void)fl;
    *n = 1;
    return cudaSuccess;
}
static cudaError_t launch(const void *f, Dim g, size_t smem, cudaStream_t s)
{
    ++launches;
    if (!g.x || !g.y || !g.z || g.x > 2147483647u || g.y > 65535 || g.z > 65535) return ret(cudaErrorInvalidConfiguration);
    if (fails(1)) return ret(cudaErrorLaunchFailure);
    if (s && ((struct stream *)s)->dev != cur) return ret(cudaErrorInvalidResourceHandle);
    if (smem > 48 * 1024 && smem > (size_t)funcs[func_at(f)].bytes[cur]) return ret(cudaErrorInvalidValue);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args)
{
    (void)args;
    return launch(f, (Dim){c->gridDim.x, c->gridDim.y, c->gridDim.z}, c->dynamicSmemBytes, c->stream);
}

static struct {
    Dim g, b;
    size_t smem;
    cudaStream_t s;
} cfg;
unsigned __cudaPushCallConfiguration(Dim g, Dim b, size_t smem, struct CUstream_st *s)
{
    cfg.g = g;
    cfg.b = b;
    cfg.smem = smem;
    cfg.s = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(Dim *g, Dim *b, size_t *smem, void *s)
{
    *g = cfg.g;
    *b = cfg.b;
    *smem = cfg.smem;
    *(cudaStream_t *)s = cfg.s;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f)
{
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, Dim g, Dim b, void **args, size_t smem, cudaStream_t s)
{
    (void)b, (void)args;
    return launch((const void *)k, g, smem, s);
}
void **__cudaRegisterFatBinary(void *f)
{
    static void *h[1];
    (void)f;
    return h;
}
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *v, char *d, const char *n, int e, size_t s, int c, int g) { (void)h, (void)v, (void)d, (void)n, (void)e, (void)s, (void)c, (void)g; }
void __cudaRegisterFunction(void **h, const char *f, char *d, const char *n, int t, void *a, void *b, void *c, void *e, int *w) { (void)h, (void)f, (void)d, (void)n, (void)t, (void)a, (void)b, (void)c, (void)e, (void)w; }
