/*
 * fake_cuda.h -- a CUDA runtime on the host, for tests of the library's host
 * code without a GPU: memory is the host's, streams and events are counters,
 * kernels do nothing unless the test's fake_kernel() does their part.  Every
 * allocation is kept with its size, the n-th from now can be made to fail
 * (fake_fail), and every memset and copy is checked against the sizes.
 */
#ifndef FAKE_CUDA_H
#define FAKE_CUDA_H

#include <cuda_runtime.h>

#include <map>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <string>

static std::map<char *, size_t> fake_allocs;
/* (the kernels' names come before this file's objects are made) */
static std::map<const void *, std::string> &fake_names()
{
    static std::map<const void *, std::string> names;
    return names;
}
static std::map<void *, float> fake_events;
static int fake_countdown;          /* allocations until one fails; 0: none does */
static size_t fake_limit;           /* device bytes there are; 0: no limit */
static size_t fake_device, fake_pinned;   /* device bytes held, pinned bytes asked for */
static int fake_bad;                /* accesses outside an allocation */
static float fake_clock;

/* the test's part of a kernel, by its name */
static void fake_kernel(const std::string &name, void **args);

static size_t fake_room(const void *p)
{
    auto it = fake_allocs.upper_bound((char *)p);
    if (it == fake_allocs.begin()) return 0;
    --it;
    const size_t at = (size_t)((char *)p - it->first);
    return at < it->second ? it->second - at : 0;
}

static cudaError_t fake_alloc(void **p, size_t n, bool device)
{
    if (fake_countdown && --fake_countdown == 0) return cudaErrorMemoryAllocation;
    if (device && fake_limit && fake_device + n > fake_limit) return cudaErrorMemoryAllocation;
    char *q = (char *)calloc(n ? n : 1, 1);
    if (!q) return cudaErrorMemoryAllocation;
    fake_allocs[q] = n;
    *(device ? &fake_device : &fake_pinned) += n;
    *p = q;
    return cudaSuccess;
}

static cudaError_t fake_release(void *p, bool device)
{
    if (!p) return cudaSuccess;
    auto it = fake_allocs.find((char *)p);
    if (it == fake_allocs.end()) {
        fake_bad++;
        return cudaErrorInvalidValue;
    }
    if (device) fake_device -= it->second;
    fake_allocs.erase(it);
    free(p);
    return cudaSuccess;
}

static cudaError_t fake_set(void *p, int v, size_t n)
{
    if (n > fake_room(p)) {
        fprintf(stderr, "memset of %zu bytes, room for %zu\n", n, fake_room(p));
        fake_bad++;
        return cudaErrorInvalidValue;
    }
    memset(p, v, n);
    return cudaSuccess;
}

static cudaError_t fake_launch(const void *f, void **args)
{
    fake_kernel(fake_names()[f], args);
    return cudaSuccess;
}

#ifndef __CUDA_ARCH__   /* the device has its own of these names */
extern "C" {
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *, dim3 *,
                            dim3 *, int *)
{
    fake_names()[f] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f)
{
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **args, size_t, cudaStream_t)
{
    return fake_launch((const void *)k, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *f, void **args)
{
    return fake_launch(f, args);
}

cudaError_t cudaMalloc(void **p, size_t n) { return fake_alloc(p, n, true); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return fake_alloc(p, n, true); }
cudaError_t cudaFree(void *p) { return fake_release(p, true); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return fake_release(p, true); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return fake_alloc(p, n, false); }
cudaError_t cudaMallocHost(void **p, size_t n) { return fake_alloc(p, n, false); }
cudaError_t cudaFreeHost(void *p) { return fake_release(p, false); }
cudaError_t cudaMemset(void *p, int v, size_t n) { return fake_set(p, v, n); }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return fake_set(p, v, n); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k)
{
    const bool to = k == cudaMemcpyHostToDevice || k == cudaMemcpyDeviceToDevice;
    const bool from = k == cudaMemcpyDeviceToHost || k == cudaMemcpyDeviceToDevice;
    if ((to && n > fake_room(d)) || (from && n > fake_room(s))) {
        fake_bad++;
        return cudaErrorInvalidValue;
    }
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t)
{
    return cudaMemcpy(d, s, n, k);
}

static cudaError_t fake_event(cudaEvent_t *e)
{
    *e = (cudaEvent_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return fake_event(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return fake_event(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t)
{
    fake_events[e] = fake_clock += 1.f;
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b)
{
    *ms = fake_events[b] - fake_events[a];
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    *s = (cudaStream_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSetAttribute(cudaStream_t, cudaStreamAttrID, const cudaStreamAttrValue *)
{
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g)
{
    *g = NULL;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long)
{
    *e = (cudaGraphExec_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e)
{
    free(e);
    return cudaSuccess;
}

cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int)
{
    *v = 1;
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *free_bytes, size_t *total)
{
    *free_bytes = *total = (size_t)1 << 38;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaDeviceSetLimit(cudaLimit, size_t) { return cudaSuccess; }
cudaError_t cudaCtxResetPersistingL2Cache(void) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *, const void *) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaPeekAtLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e)
{
    return e == cudaErrorMemoryAllocation ? "out of memory" : "error";
}

void fake_fail(int n) { fake_countdown = n; }
void fake_have(size_t bytes) { fake_limit = bytes; }
size_t fake_held(void) { return fake_device; }
size_t fake_pinned_bytes(void) { return fake_pinned; }
int fake_errors(void) { return fake_bad; }
}
#endif

#endif
