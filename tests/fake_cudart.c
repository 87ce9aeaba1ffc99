/* A stand-in for the CUDA runtime, preloaded by tests of the library's host code
 * (no GPU, no kernel runs). Device memory is host memory. It models what ordering
 * tests need: a copy from pageable memory or a memset on one stream may still be
 * pending when the call returns, so a launch on another (non-blocking) stream
 * before a synchronisation is counted as unordered. */
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

static cudaError_t last;
static int live, mallocs_until_failure = -1, launches, unordered, instantiated;
static char pending[64]; /* by stream number; 0: the legacy stream */
static int streams;
static struct {
    char* at;
    size_t bytes;
} block[256]; /* live allocations */
/* address space that a program has reserved, of which it has mapped the first part */
static char* reserved;
static size_t reserved_bytes, mapped_bytes;

void fake_fail_malloc(int n) { mallocs_until_failure = n; } /* the n-th from now, 0 the next */
int fake_live_allocations(void) { return live; }
int fake_launches(void) { return launches; }
int fake_unordered_launches(void) { return unordered; }
void fake_reserve(void* at, size_t bytes, size_t mapped)
{
    reserved       = at;
    reserved_bytes = bytes;
    mapped_bytes   = mapped;
}
/* the first words of the last solve launch's arguments (its SolveGeom) */
static int solve[30];
void fake_last_solve(int* words) { memcpy(words, solve, sizeof(solve)); }
int fake_graphs_instantiated(void) { return instantiated; }

static int number(cudaStream_t s) { return (int)(size_t)s; }

cudaError_t cudaGetLastError(void)
{
    cudaError_t e = last;
    last          = cudaSuccess;
    return e;
}
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d)
{
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(struct cudaDeviceProp* p, int d)
{
    (void)d;
    memset(p, 0, sizeof(*p));
    strcpy(p->name, "fake GPU");
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n)
{
    if (mallocs_until_failure >= 0 && mallocs_until_failure-- == 0) {
        *p = NULL;
        return last = cudaErrorMemoryAllocation;
    }
    int b = 0;
    while (block[b].at)
        ++b;
    ++live;
    *p = block[b].at = calloc(1, n ? n : 1);
    block[b].bytes   = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    for (int b = 0; p && b < 256; ++b)
        if (block[b].at == p) {
            block[b].at = NULL;
            --live;
        }
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n)
{
    memset(p, v, n);
    pending[0] = 1;
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s)
{
    memset(p, v, n);
    pending[number(s)] = 1;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k)
{
    memcpy(d, s, n);
    pending[0] = k == cudaMemcpyHostToDevice;
    return cudaSuccess;
}
/* whether a range starts in the reservation and leaves what is mapped */
static int outside(const void* p, size_t n)
{
    const char* a = p;
    return a >= reserved && a < reserved + reserved_bytes && a + n > reserved + mapped_bytes;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k,
                            cudaStream_t st)
{
    (void)k;
    if (outside(d, n) || outside(s, n))
        return last = cudaErrorInvalidValue;
    memcpy(d, s, n);
    pending[number(st)] = 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { memset(pending, 0, sizeof(pending)); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { pending[number(s)] = 0; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f)
{
    (void)f;
    *s = (cudaStream_t)(size_t)++streams;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int p)
{
    (void)p;
    return cudaStreamCreateWithFlags(s, f);
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) { *lo = *hi = 0; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f)
{
    (void)s, (void)e, (void)f;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e, (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
/* each interval is shorter than the one before it, so a tuner keeps its last candidate */
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b)
{
    static float t = 1e6f;
    (void)a, (void)b;
    *ms = t -= 1.0f;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v)
{
    (void)f, (void)a, (void)v;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* f)
{
    (void)f;
    memset(a, 0, sizeof(*a));
    a->numRegs = 255;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int b, size_t s)
{
    (void)f, (void)b, (void)s;
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b,
                                                                   size_t s, unsigned flags)
{
    (void)flags;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, f, b, s);
}
static int encode(void) { return 0; }
static CUresult address_range(CUdeviceptr* base, size_t* bytes, CUdeviceptr p)
{
    const char* a = (const char*)(uintptr_t)p;
    if (a >= reserved && a < reserved + mapped_bytes) {
        *base  = (CUdeviceptr)(uintptr_t)reserved;
        *bytes = mapped_bytes;
        return CUDA_SUCCESS;
    }
    for (int b = 0; b < 256; ++b)
        if (block[b].at && a >= block[b].at && a < block[b].at + block[b].bytes) {
            *base  = (CUdeviceptr)(uintptr_t)block[b].at;
            *bytes = block[b].bytes;
            return CUDA_SUCCESS;
        }
    return CUDA_ERROR_NOT_FOUND;
}
static CUresult attributes(unsigned n, CUpointer_attribute* what, void** to, CUdeviceptr p)
{
    const char* a  = (const char*)(uintptr_t)p;
    const int vm   = a >= reserved && a < reserved + reserved_bytes;
    CUdeviceptr at = (CUdeviceptr)(uintptr_t)reserved;
    size_t bytes   = reserved_bytes;
    const int gpu  = address_range(&at, &bytes, p) == CUDA_SUCCESS;
    if (vm) { /* RANGE_* tell of the reservation, not of what is mapped */
        at    = (CUdeviceptr)(uintptr_t)reserved;
        bytes = reserved_bytes;
    }
    for (unsigned i = 0; i < n; ++i)
        switch (what[i]) {
        case CU_POINTER_ATTRIBUTE_MEMORY_TYPE: *(unsigned*)to[i] = gpu ? CU_MEMORYTYPE_DEVICE : 0; break;
        case CU_POINTER_ATTRIBUTE_IS_MANAGED: *(unsigned*)to[i] = 0; break;
        case CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL: *(int*)to[i] = gpu ? 0 : -2; break;
        case CU_POINTER_ATTRIBUTE_IS_LEGACY_CUDA_IPC_CAPABLE: *(unsigned*)to[i] = gpu && !vm; break;
        case CU_POINTER_ATTRIBUTE_MEMPOOL_HANDLE: *(void**)to[i] = NULL; break;
        case CU_POINTER_ATTRIBUTE_RANGE_START_ADDR: *(CUdeviceptr*)to[i] = gpu ? at : 0; break;
        case CU_POINTER_ATTRIBUTE_RANGE_SIZE: *(size_t*)to[i] = gpu ? bytes : 0; break;
        default: return CUDA_ERROR_INVALID_VALUE;
        }
    return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPoint(const char* name, void** fn, unsigned long long flags,
                                    enum cudaDriverEntryPointQueryResult* q)
{
    (void)flags;
    *fn = strcmp(name, "cuTensorMapEncodeTiled") == 0   ? (void*)encode
          : strcmp(name, "cuPointerGetAttributes") == 0 ? (void*)attributes
          : strcmp(name, "cuMemGetAddressRange") == 0   ? (void*)address_range
                                                        : NULL;
    *q  = *fn ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
static cudaError_t launch(cudaStream_t st)
{
    ++launches;
    for (int s = 0; s < (int)sizeof(pending); ++s)
        if (pending[s] && s != number(st)) {
            ++unordered;
            break;
        }
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t smem, cudaStream_t s)
{
    (void)f, (void)g, (void)b, (void)args, (void)smem;
    return launch(s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args)
{
    (void)f;
    if (c->dynamicSmemBytes > 0)
        memcpy(solve, args[1], sizeof(solve));
    return launch(c->stream);
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m)
{
    (void)s, (void)m;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g)
{
    (void)s;
    *g = (cudaGraph_t)1;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long f)
{
    (void)g, (void)f;
    *e = (cudaGraphExec_t)(size_t)++instantiated;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s)
{
    (void)e, (void)s;
    return cudaSuccess;
}
