/* A CUDA runtime for the core's host code on a machine without a GPU: device
 * memory is host memory, and every call is done when it returns, except the
 * copies and clears that CUDA lets outlive their call on the legacy stream
 * (fake_pending below).  Included by one source file of a test program that
 * also includes the host code itself; the kernel launches are the test's.
 *
 * Blocks come from slots of one size, so that a test can decide which address
 * an allocation gets (fake_pick); a new block holds 0xAB. */
#pragma once

#include <cuda_runtime.h>
#include <sys/mman.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#define CHECK_THAT(cond, ...)                                     \
    do {                                                          \
        if (!(cond)) {                                            \
            fprintf(stderr, "%s:%d: ", __FILE__, __LINE__);       \
            fprintf(stderr, __VA_ARGS__);                         \
            fprintf(stderr, "\n");                                \
            exit(1);                                              \
        }                                                         \
    } while (0)

static constexpr size_t kSlot = (size_t)512 << 20;
static constexpr int kSlots = 128;
static char *fake_base;
static bool fake_used[kSlots];
/* an address for an allocation of `bytes` (pinned: host memory), or NULL */
static std::function<void *(size_t bytes, bool pinned)> fake_pick;
/* allocations that succeed before one fails (-1: none fails) */
static int fake_fail_after = -1;
/* legacy-stream work that may still be under way when its call returns:
 * copies from pageable memory to the device and clears.  Done by a wait for
 * the device or for the legacy stream. */
static std::vector<std::function<void()>> fake_pending;

static int slot_of(const void *p) { return (int)(((const char *)p - fake_base) / (ptrdiff_t)kSlot); }
static bool fake_is_block(const void *p)
{
    return fake_base && (const char *)p >= fake_base && (const char *)p < fake_base + kSlot * kSlots;
}

static void *fake_alloc(size_t bytes, bool pinned)
{
    if (!fake_base) {
        void *m = mmap(nullptr, kSlot * kSlots, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE,
                       -1, 0);
        CHECK_THAT(m != MAP_FAILED, "mmap");
        fake_base = (char *)m;
    }
    CHECK_THAT(bytes <= kSlot, "a block of %zu bytes", bytes);
    void *p = fake_pick ? fake_pick(bytes, pinned) : nullptr;
    for (int i = 0; !p && i < kSlots; i++)
        if (!fake_used[i])
            p = fake_base + kSlot * i;
    CHECK_THAT(p && !fake_used[slot_of(p)], "no slot");
    fake_used[slot_of(p)] = true;
    memset(p, 0xAB, bytes < ((size_t)8 << 20) ? bytes : (size_t)8 << 20);
    return p;
}

static void fake_run_pending()
{
    for (auto &f : fake_pending)
        f();
    fake_pending.clear();
}

extern "C" {
static cudaError_t fake_alloc_to(void **p, size_t n, bool pinned)
{
    if (fake_fail_after == 0)
        return cudaErrorMemoryAllocation;
    if (fake_fail_after > 0)
        fake_fail_after--;
    *p = fake_alloc(n, pinned);
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return fake_alloc_to(p, n, false); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return fake_alloc_to(p, n, true); }
cudaError_t cudaMallocHost(void **p, size_t n) { return fake_alloc_to(p, n, true); }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaFree(void *p)
{
    if (p) {
        fake_run_pending();
        CHECK_THAT(fake_is_block(p) && fake_used[slot_of(p)], "free of a block that is not held");
        fake_used[slot_of(p)] = false;
    }
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k)
{
    if (k == cudaMemcpyHostToDevice && !fake_is_block(s)) {
        std::vector<char> staged((const char *)s, (const char *)s + n);
        fake_pending.push_back([=] { memcpy(d, staged.data(), n); });
    } else {
        fake_run_pending();
        memcpy(d, s, n);
    }
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n)
{
    fake_pending.push_back([=] { memset(d, v, n); });
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { fake_run_pending(); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    if (!s || s == cudaStreamLegacy)
        fake_run_pending();
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.1f; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int)   /* _v2 by the header's macro */
{
    memset(p, 0, sizeof(*p));
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
}
