// Stand-in for the CUDA runtime API used by the context's host code
// (luthe_b200/csrc/api.cu), so that it can be compiled and exercised on a
// machine without a GPU (test infrastructure only).  Memory is host memory.
// Streams and events carry what is known to be ordered before them, so that
// the harness can tell whether two uses of one buffer are ordered.
#pragma once
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>
#include <map>
#include <set>
#include <vector>

#define __device__
#define __align__(x) __attribute__((aligned(x)))

typedef int cudaError_t;
enum {
    cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2, cudaErrorCooperativeLaunchTooLarge = 720,
    cudaErrorNotSupported = 801,
    cudaErrorStreamCaptureIsolation = 906, cudaErrorCapturedEvent = 907
};
struct fake_graph {
    std::vector<const void *> uses;  // buffers of the captured launches
    std::map<const void *, std::set<int>> ops;
};
struct fake_stream {
    std::set<int> before;            // operations ordered before whatever comes next
    fake_graph *capture = nullptr;   // capturing into
    bool caller = false;             // ... for the caller, not for the context
    bool limited = false;            // to some of the SMs
};
struct fake_event {
    std::set<int> before;
    fake_graph *capture = nullptr;   // recorded during a capture
};
typedef fake_stream *cudaStream_t;
typedef fake_event *cudaEvent_t;
typedef fake_graph *cudaGraph_t, *cudaGraphExec_t;
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone = 0, cudaStreamCaptureStatusActive = 1 };
enum cudaStreamCaptureMode { cudaStreamCaptureModeThreadLocal = 1 };
enum cudaDeviceAttr { cudaDevAttrMaxSharedMemoryPerMultiprocessor, cudaDevAttrCooperativeLaunch };
#define cudaStreamNonBlocking 1
#define cudaEventDisableTiming 2
struct cudaDeviceProp {
    char name[256];
    int major, minor, multiProcessorCount;
};

struct FakeCuda {
    fake_stream legacy;
    int ops = 0;                             // operations enqueued so far
    std::map<const void *, std::set<int>> uses;  // of each shared buffer
    int races = 0;                           // uses of a buffer not ordered after an earlier one
    std::map<int, int> fail_malloc;          // n-th allocation from now -> error
};
static FakeCuda g_fake;
static inline fake_stream *fake_of(cudaStream_t s) { return s ? s : &g_fake.legacy; }

// one operation on stream s that uses the given shared buffer
static inline void fake_use(const void *buf, cudaStream_t s)
{
    fake_stream *st = fake_of(s);
    if (st->capture) st->capture->uses.push_back(buf);
    std::set<int> &uses = st->capture ? st->capture->ops[buf] : g_fake.uses[buf];
    for (int op : uses) g_fake.races += !st->before.count(op);
    const int op = g_fake.ops++;
    uses.insert(op);
    st->before.insert(op);
}

static inline const char *cudaGetErrorString(cudaError_t) { return "fake"; }
static inline cudaError_t cudaGetLastError() { return cudaSuccess; }
static inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
static inline cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int)
{
    strcpy(p->name, "fake");
    p->major = 10;
    p->minor = 0;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
static inline cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrCooperativeLaunch ? 1 : 233472;
    return cudaSuccess;
}
static inline cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
static inline cudaError_t cudaMalloc(void **p, size_t bytes)
{
    std::map<int, int> next;
    int rc = cudaSuccess;
    for (auto &f : g_fake.fail_malloc)
        if (f.first == 0) rc = f.second;
        else next[f.first - 1] = f.second;
    g_fake.fail_malloc.swap(next);
    if (rc != cudaSuccess) return rc;
    *p = calloc(1, bytes);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
static inline cudaError_t cudaFree(void *p)
{
    g_fake.uses.clear();  // waits for the device
    free(p);
    return cudaSuccess;
}
static inline cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind)
{
    memcpy(d, s, n);
    return cudaSuccess;
}
static inline cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    memcpy(d, s, n);
    return cudaSuccess;
}
static inline cudaError_t cudaMemset(void *d, int v, size_t n)
{
    memset(d, v, n);
    return cudaSuccess;
}
static inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    *s = new fake_stream;
    return cudaSuccess;
}
static inline cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    delete s;
    return cudaSuccess;
}
static inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
static inline cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *st)
{
    *st = fake_of(s)->capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
static inline cudaError_t cudaStreamGetCaptureInfo(cudaStream_t s, cudaStreamCaptureStatus *st, unsigned long long *id)
{
    *id = (unsigned long long)(size_t)fake_of(s)->capture;
    return cudaStreamIsCapturing(s, st);
}
static inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    *e = new fake_event;
    return cudaSuccess;
}
static inline cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
static inline cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    delete e;
    return cudaSuccess;
}
static inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
static inline cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t)
{
    *ms = 1.f;
    return cudaSuccess;
}
static inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    e->capture = fake_of(s)->capture;
    e->before = fake_of(s)->before;
    return cudaSuccess;
}
static inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
    if (fake_of(s)->capture != e->capture) return e->capture ? cudaErrorCapturedEvent : cudaErrorStreamCaptureIsolation;
    fake_of(s)->before.insert(e->before.begin(), e->before.end());
    return cudaSuccess;
}
static inline cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode)
{
    s->capture = new fake_graph;
    s->caller = false;
    return cudaSuccess;
}
static inline cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g)
{
    *g = s->capture;
    s->capture = nullptr;
    return cudaSuccess;
}
static inline cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, unsigned long long)
{
    *e = new fake_graph(*g);
    return cudaSuccess;
}
static inline cudaError_t cudaGraphDestroy(cudaGraph_t g)
{
    delete g;
    return cudaSuccess;
}
static inline cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g)
{
    delete g;
    return cudaSuccess;
}
static inline cudaError_t cudaGraphLaunch(cudaGraphExec_t g, cudaStream_t s)
{
    for (const void *b : g->uses) fake_use(b, s);
    return cudaSuccess;
}
template <typename T>
static inline cudaError_t cudaGetSymbolAddress(void **p, T &symbol)
{
    *p = (void *)&symbol;
    return cudaSuccess;
}
