/*
 * st_xfer.cu -- copies between device memory and the caller's host arrays.
 *
 * The explicit API takes plain host memory.  A cudaMemcpy to or from pageable memory stages
 * through the driver's own buffers on one host thread: 13 to 17 GB/s over a link that moves
 * 50 GB/s from pinned memory, and 4.5 GB/s into freshly allocated arrays, whose pages that one
 * thread faults in.  Here the copy is cut into pieces of XFER_PIECE bytes; a few host threads
 * take pieces in turn, and each moves its piece through a pinned buffer of its own: the copies
 * of one direction queue on the link while other threads copy to or from the caller's memory
 * (and fault its pages).  Measured on one B200 host (16 hardware threads), whole API calls:
 * 1e6 parcels with four steps and owning cells read back 14.0 -> 3.9 ms, 1e7 parcels set
 * 162 -> 30 ms, an adjoint pass with 124 MB in and out 18.6 -> 10.7 ms, a 64^3 coupled step
 * with double fields 0.78 -> 0.75 ms.
 *
 * The staging buffer belongs to the process: a pinned piece for each thread that a copy has work
 * for, at most XFER_THREADS (24 MB), made when a copy first needs it and freed with the last
 * handle.  Pinning is dear (16 ms for 24 MB, 2.5 ms to free), so copies go through plain
 * cudaMemcpyAsync until XFER_RENT bytes have been copied: a program of small copies, or of one
 * small handle after another, does not pay for it each time (a fresh handle's 1e5 FP64 parcels set
 * 23 ms when the first copy of 2 MB made the buffer, 3.0 ms now, the handle destroyed 5.9 and
 * 2.8 ms).  Staging earns 0.04 ms per MB up and 0.16 down into pages that are used again, so a
 * later line (128 MB) suits fresh handles of 1e6 parcels in turn (set 12 ms, 28 with this line), and
 * a program with more to copy pays for it then, in a pass (1e6 parcels' first adjoint pass on a
 * fresh handle 27 to 35 ms, 11 with this line).  One copy uses the buffer at a time; a copy that
 * finds it taken (another host thread's), or cannot have it, and copies to pinned memory or below
 * XFER_MIN, go through plain cudaMemcpyAsync, and so do those of a handle in a context other than
 * the device's primary one.
 */
#include <algorithm>
#include <atomic>
#include <cstring>
#include <cstdint>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include "st_xfer.h"

namespace st {
namespace {

/* 2 MB pieces (1 MB: 1e6 parcels read back in 2.90 against 2.37 ms; 256 KB 3.5 ms), 1 MB below
 * 16 MB in all (three 2 MB pieces would leave threads without one: a 64^3 coupled step 0.81
 * against 0.70 ms).  Twelve threads against eight: 50 MB into fresh pages 3.43 -> 3.02 ms,
 * sixteen 3.74 ms. */
constexpr size_t XFER_PIECE = (size_t)2 << 20;
constexpr size_t XFER_MIN = (size_t)2 << 20;
constexpr size_t XFER_RENT = (size_t)48 << 20;
constexpr int XFER_THREADS = 12;

std::mutex g_users_mu;
int g_users = 0;             /* live handles */
std::mutex g_pin_mu;         /* held by the copy that uses the buffer */
unsigned char* g_pin = nullptr;   /* [g_pieces][XFER_PIECE], pinned */
int g_pieces = 0;
size_t g_copied = 0;         /* bytes copied since the buffer was last given back */

struct Piece {
    unsigned char* host;
    unsigned char* dev;
    size_t bytes;
};

cudaError_t plain(const XferSeg* seg, int n, bool down, cudaStream_t s)
{
    for (int k = 0; k < n; ++k) {
        if (!seg[k].bytes) continue;
        const cudaError_t e =
            down ? cudaMemcpyAsync(seg[k].host, seg[k].dev, seg[k].bytes, cudaMemcpyDeviceToHost, s)
                 : cudaMemcpyAsync(seg[k].dev, seg[k].host, seg[k].bytes, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) return e;
    }
    return cudaStreamSynchronize(s);
}

/* Whether the device's primary context is current on this thread.  The staging buffers and the
 * helper threads (cudaSetDevice) are the primary context's; a caller that made its handle in a
 * context of its own (driver API) has its copies on its own thread. */
bool primary_current(int device)
{
    using DeviceGet = int (*)(int*, int);
    using GetCurrent = int (*)(void**);
    using GetState = int (*)(int, unsigned*, int*);
    using Retain = int (*)(void**, int);
    using Release = int (*)(int);
    struct Api {
        DeviceGet device = nullptr;
        GetCurrent current = nullptr;
        GetState state = nullptr;
        Retain retain = nullptr;
        Release release = nullptr;
        static void* find(const char* name)
        {
            void* f = nullptr;
            cudaDriverEntryPointQueryResult r;
            if (cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &r) != cudaSuccess ||
                r != cudaDriverEntryPointSuccess) {
                cudaGetLastError();
                return nullptr;
            }
            return f;
        }
        Api()
        {
            device = reinterpret_cast<DeviceGet>(find("cuDeviceGet"));
            current = reinterpret_cast<GetCurrent>(find("cuCtxGetCurrent"));
            state = reinterpret_cast<GetState>(find("cuDevicePrimaryCtxGetState"));
            retain = reinterpret_cast<Retain>(find("cuDevicePrimaryCtxRetain"));
            release = reinterpret_cast<Release>(find("cuDevicePrimaryCtxRelease"));
        }
    };
    static const Api api;
    if (!api.device || !api.current || !api.state || !api.retain || !api.release) return false;
    void *now = nullptr, *primary = nullptr;
    unsigned flags = 0;
    int dev = 0, active = 0;
    /* (retaining an inactive primary context would make it) */
    if (api.device(&dev, device) || api.current(&now) || api.state(dev, &flags, &active) ||
        !active || api.retain(&primary, dev))
        return false;
    api.release(dev);
    return now == primary;
}

/* Takes pieces from the shared counter until none is left or a copy failed.  `helper`: on a
 * thread of its own, which first needs the device; where it does not get it, or cannot work on
 * the stream, it leaves the pieces to the others. */
void worker(const std::vector<Piece>& pieces, std::atomic<size_t>& next, std::atomic<int>& err,
            unsigned char* pin, bool down, int device, cudaStream_t s, bool helper)
{
    cudaEvent_t ev = nullptr;
    cudaError_t e = cudaSuccess;
    if (helper) {
        /* what its copies may do is the caller's affair, not a capture's on another thread */
        cudaStreamCaptureMode relaxed = cudaStreamCaptureModeRelaxed;
        if (cudaThreadExchangeStreamCaptureMode(&relaxed) != cudaSuccess ||
            cudaSetDevice(device) != cudaSuccess)
            return;
    }
    e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (helper && (e != cudaSuccess || cudaEventRecord(ev, s) != cudaSuccess)) {
        if (ev) cudaEventDestroy(ev);
        return;
    }
    while (e == cudaSuccess && err.load() == (int)cudaSuccess) {
        const size_t k = next.fetch_add(1);
        if (k >= pieces.size()) break;
        const Piece& p = pieces[k];
        if (!down) memcpy(pin, p.host, p.bytes);
        e = down ? cudaMemcpyAsync(pin, p.dev, p.bytes, cudaMemcpyDeviceToHost, s)
                 : cudaMemcpyAsync(p.dev, pin, p.bytes, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaEventRecord(ev, s);
        if (e == cudaSuccess) e = cudaEventSynchronize(ev);   /* the buffer is free again */
        if (e == cudaSuccess && down) memcpy(p.host, pin, p.bytes);
    }
    if (ev) cudaEventDestroy(ev);
    if (e != cudaSuccess) {
        int ok = (int)cudaSuccess;
        err.compare_exchange_strong(ok, (int)e);
    }
}

/* Pinned memory is copied to and from directly. */
bool pinned(const void* p)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type != cudaMemoryTypeUnregistered;
}

void give_back()
{
    if (g_pin) cudaFreeHost(g_pin);
    g_pin = nullptr;
    g_pieces = 0;
}

/* Pinned pieces for nt threads, or for as many as there are when no more can be had. */
int have_pieces(int nt)
{
    if (g_pin && !pinned(g_pin)) {        /* gone with a reset device */
        g_pin = nullptr;
        g_pieces = 0;
    }
    if (g_pieces >= nt) return nt;
    void* p = nullptr;
    if (cudaHostAlloc(&p, nt * XFER_PIECE, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return g_pieces;
    }
    give_back();
    g_pin = static_cast<unsigned char*>(p);
    return g_pieces = nt;
}

cudaError_t xfer(const XferSeg* seg, int n, bool down, int device, cudaStream_t s,
                 size_t ahead)
{
    size_t total = 0;
    bool pageable = false;
    for (int k = 0; k < n; ++k) total += seg[k].bytes;
    if (total >= XFER_MIN)
        for (int k = 0; k < n; ++k) pageable = pageable || !pinned(seg[k].host);
    std::unique_lock<std::mutex> lk(g_pin_mu, std::defer_lock);
    /* (the per-thread stream is another one on every thread) */
    if (!pageable || s == cudaStreamPerThread || !primary_current(device) || !lk.try_lock())
        return plain(seg, n, down, s);
    g_copied += total;
    if (g_copied + ahead < XFER_RENT) return plain(seg, n, down, s);
    const int cores = (int)std::thread::hardware_concurrency();
    int nt = (int)(total / XFER_MIN) + 1;      /* a thread costs about 20 us: 1 MB each at least */
    if (nt > XFER_THREADS) nt = XFER_THREADS;
    if (cores > 0 && nt > cores) nt = cores;
    if ((nt = have_pieces(nt)) == 0) return plain(seg, n, down, s);
    const size_t piece = total >= 8 * XFER_PIECE ? XFER_PIECE : XFER_PIECE / 2;
    std::vector<Piece> pieces;
    std::vector<std::thread> ts;
    try {
        pieces.reserve(total / piece + n);
        ts.reserve(nt);
    } catch (const std::bad_alloc&) {
        return plain(seg, n, down, s);
    }
    for (int k = 0; k < n; ++k) {
        unsigned char* hp = static_cast<unsigned char*>(seg[k].host);
        unsigned char* dp = static_cast<unsigned char*>(seg[k].dev);
        for (size_t o = 0; o < seg[k].bytes; o += piece) {
            const size_t b = std::min(seg[k].bytes - o, piece);
            pieces.push_back({hp + o, dp + o, b});
        }
    }
    std::atomic<size_t> next{0};
    std::atomic<int> err{(int)cudaSuccess};
    for (int t = 1; t < nt; ++t) {
        try {
            ts.emplace_back(worker, std::cref(pieces), std::ref(next), std::ref(err),
                            g_pin + t * XFER_PIECE, down, device, s, true);
        } catch (...) {
            break;                             /* no more threads: fewer take the pieces */
        }
    }
    worker(pieces, next, err, g_pin, down, device, s, false);
    for (std::thread& t : ts) t.join();
    if (err.load() != (int)cudaSuccess) cudaStreamSynchronize(s);   /* no copy left in flight */
    return (cudaError_t)err.load();
}

}  // namespace

cudaError_t xfer_down(const XferSeg* seg, int n, int device, cudaStream_t s, size_t ahead)
{
    return xfer(seg, n, true, device, s, ahead);
}

cudaError_t xfer_up(const XferSeg* seg, int n, int device, cudaStream_t s, size_t ahead)
{
    return xfer(seg, n, false, device, s, ahead);
}

void xfer_retain()
{
    std::lock_guard<std::mutex> lk(g_users_mu);
    ++g_users;
}

void xfer_release()
{
    std::lock_guard<std::mutex> lk(g_users_mu);
    if (--g_users > 0) return;
    std::lock_guard<std::mutex> pin(g_pin_mu);
    give_back();
    g_copied = 0;
}

}  // namespace st
