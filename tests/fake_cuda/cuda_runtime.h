/* A stand-in for the CUDA runtime calls of st_xfer.cu, for tests on the CPU: device memory is host
 * memory, streams and events are words, and every call is counted. */
#ifndef FAKE_CUDA_RUNTIME_H
#define FAKE_CUDA_RUNTIME_H

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <set>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2,
                   cudaErrorInvalidResourceHandle = 400, cudaErrorUnknown = 999 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost };
enum cudaMemoryType { cudaMemoryTypeUnregistered, cudaMemoryTypeHost };
enum cudaStreamCaptureMode { cudaStreamCaptureModeGlobal, cudaStreamCaptureModeThreadLocal,
                             cudaStreamCaptureModeRelaxed };
enum cudaDriverEntryPointQueryResult { cudaDriverEntryPointSuccess };
struct cudaPointerAttributes { cudaMemoryType type; };
typedef int* cudaStream_t;
typedef int* cudaEvent_t;
#define cudaStreamPerThread ((cudaStream_t)0x2)
#define cudaEventDisableTiming 2
#define cudaHostAllocPortable 1
#define cudaEnableDefault 0

namespace fake {
extern std::atomic<int> set_device, host_allocs, copies, syncs;
extern std::atomic<long> host_bytes;
extern thread_local void* context;          /* current on the thread */
extern thread_local int mode;
extern void *primary, *stream_context;
extern bool refuse_alloc;
extern int global_capture;                  /* a capture in global mode runs on some thread */
extern std::atomic<int> fail_copy;          /* the copy that fails (counted from 1), 0: none */
extern std::mutex mu;
extern std::set<void*> pinned;
inline bool unsafe() { return global_capture && mode != cudaStreamCaptureModeRelaxed; }
inline int device_get(int* d, int ordinal) { *d = ordinal; return 0; }
inline int get_current(void** c) { *c = context; return 0; }
inline int get_state(int, unsigned* f, int* a) { *f = 0; *a = primary != nullptr; return 0; }
inline int retain(void** c, int) { *c = primary; return 0; }
inline int release(int) { return 0; }
}  // namespace fake

inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaSetDevice(int)
{
    ++fake::set_device;
    fake::context = fake::primary;
    return cudaSuccess;
}
inline cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m)
{
    const int old = fake::mode;
    fake::mode = *m;
    *m = (cudaStreamCaptureMode)old;
    return cudaSuccess;
}
inline cudaError_t cudaGetDriverEntryPoint(const char* n, void** f, unsigned long long,
                                           cudaDriverEntryPointQueryResult* r)
{
    *r = cudaDriverEntryPointSuccess;
    *f = !strcmp(n, "cuDeviceGet")                  ? (void*)fake::device_get
         : !strcmp(n, "cuCtxGetCurrent")            ? (void*)fake::get_current
         : !strcmp(n, "cuDevicePrimaryCtxGetState") ? (void*)fake::get_state
         : !strcmp(n, "cuDevicePrimaryCtxRetain")   ? (void*)fake::retain
                                                    : (void*)fake::release;
    return cudaSuccess;
}
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    if (fake::refuse_alloc || fake::unsafe()) return cudaErrorMemoryAllocation;
    *p = malloc(n);
    ++fake::host_allocs;
    fake::host_bytes += (long)n;
    std::lock_guard<std::mutex> lk(fake::mu);
    fake::pinned.insert(*p);
    return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p)
{
    std::lock_guard<std::mutex> lk(fake::mu);
    if (!fake::pinned.erase(p)) return cudaErrorInvalidValue;
    free(p);
    return cudaSuccess;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    std::lock_guard<std::mutex> lk(fake::mu);
    a->type = fake::pinned.count((void*)p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    if (fake::context != fake::stream_context) return cudaErrorInvalidResourceHandle;
    if (++fake::copies == fake::fail_copy) return cudaErrorUnknown;
    memcpy(d, s, n);
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    ++fake::syncs;
    return fake::context == fake::stream_context ? cudaSuccess : cudaErrorInvalidResourceHandle;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
    *e = new int(0);
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    delete e;
    return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t)
{
    return fake::context == fake::stream_context ? cudaSuccess : cudaErrorInvalidResourceHandle;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t)
{
    return fake::unsafe() ? cudaErrorUnknown : cudaSuccess;
}

#endif
