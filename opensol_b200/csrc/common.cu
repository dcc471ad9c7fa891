// Thread-local error message and the library-wide entry points of opensol_fdtd.h.
#include "common.cuh"

#include <sys/mman.h>
#include <unistd.h>

#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

namespace os {

static thread_local std::string g_last_error;

void set_error(const char *fmt, ...) {
    char buf[1024];
    va_list args;
    va_start(args, fmt);
    vsnprintf(buf, sizeof(buf), fmt, args);
    va_end(args);
    g_last_error = buf;
}

const std::string &last_error() { return g_last_error; }

int cuda_status(cudaError_t err, const char *what) {
    set_error("%s failed: %s (%s)", what, cudaGetErrorName(err), cudaGetErrorString(err));
    if (err == cudaErrorMemoryAllocation) return OS_ERR_NO_MEMORY;
    return OS_ERR_CUDA;
}

// ---- device memory pool

struct PoolEvents {
    std::vector<cudaEvent_t> events;
    int refs = 0;   // pooled blocks still waiting on them, plus the releaser until pool_events_done
};

namespace {
struct PoolBlock {
    void *ptr;
    PoolEvents *events;
};
std::mutex g_pool_mutex;
std::map<std::pair<int, size_t>, std::vector<PoolBlock>> g_pool;   // (device, class) -> blocks, last in first out
size_t g_pool_bytes = 0;
constexpr size_t kPoolLimit = (size_t)16 << 30;   // bytes kept per process; beyond it a released block is freed

// drop one reference (g_pool_mutex held); the last one destroys the events
void unref(PoolEvents *e) {
    if (e && --e->refs == 0) {
        for (cudaEvent_t ev : e->events) cudaEventDestroy(ev);
        delete e;
    }
}
}  // namespace

size_t pool_class(size_t bytes) {
    // 1/8-octave classes above 2 KiB (at most 12.5 % slack), multiples of 256 bytes below
    if (bytes <= 2048) return (bytes + 255) / 256 * 256;
    size_t p = 2048;
    while (p * 2 <= bytes) p *= 2;   // p <= bytes < 2 p
    const size_t step = p / 8;
    return (bytes + step - 1) / step * step;
}

PoolEvents *pool_events(const cudaStream_t *streams, int n) {
    PoolEvents *e = new PoolEvents();
    for (int k = 0; k < n; ++k) {
        cudaEvent_t ev;
        if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) continue;
        if (cudaEventRecord(ev, streams[k]) != cudaSuccess) {
            cudaEventDestroy(ev);
            continue;
        }
        e->events.push_back(ev);
    }
    e->refs = 1;
    return e;
}

void pool_events_done(PoolEvents *events) {
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    unref(events);
}

void pool_give(int device, void *ptr, size_t cls, PoolEvents *events) {
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (g_pool_bytes + cls > kPoolLimit) {
        // over the limit: free it (cudaFree orders itself after the device's work)
        cudaFree(ptr);
        return;
    }
    if (events) ++events->refs;
    g_pool[{device, cls}].push_back(PoolBlock{ptr, events});
    g_pool_bytes += cls;
}

void *pool_take(int device, size_t cls) {
    PoolBlock b{nullptr, nullptr};
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        auto it = g_pool.find({device, cls});
        if (it == g_pool.end() || it->second.empty()) return nullptr;
        b = it->second.back();
        it->second.pop_back();
        g_pool_bytes -= cls;
    }
    // the previous owner's last work on the block has finished before it is handed out again
    if (b.events)
        for (cudaEvent_t ev : b.events->events) cudaEventSynchronize(ev);
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        unref(b.events);
    }
    return b.ptr;
}

// ---- device-to-host reads
//
// A read into ordinary memory goes through the driver's staging buffer and one core, which also takes the page faults
// of a fresh array: 4.7 GB/s (805 MB of 8192 x 8192 fields in 170 ms).  A large read is cut into chunks that several
// threads fetch into page-locked slots of their own, two each, and copy out while the next chunk travels.  The copies
// go on a stream of the reader's own, behind the caller's stream by an event recorded in the calling thread: another
// thread may not use the caller's handle (cudaStreamPerThread names a different stream in each).  The slots and streams
// are made once per process (and device), used by one read at a time (another read meanwhile takes the plain copy) and
// freed by pool_trim.  Memory that the driver copies to directly (page-locked, managed) takes one plain copy.
namespace {
constexpr size_t kReadChunk = (size_t)2 << 20;
constexpr int kReadThreads = 8;
// Below these the threads cost more than they save: into pages not there yet (a fresh array: the copying core also takes
// their faults, 2 GB/s) and into pages that are.  Measured, us for one plain copy and for the threads: 4.9 MB fresh 2550
// and 2430, there 290-460 and 540-600; 7.9 MB 4050 and 2700, 425-670 and 620-760; 15.8 MB 8100 and 3500, 800-1250 and
// 930-1080; 23.8 MB 12000 and 4100, 1160-1930 and 980-1320; 31.8 MB 16000 and 5000, 1560-2850 and 1180-1600.
constexpr size_t kReadMin = (size_t)4 << 20, kReadMinResident = (size_t)24 << 20;
std::mutex g_read_mutex;
unsigned char *g_read_slots = nullptr;   // kReadThreads x 2 chunks, page-locked
cudaStream_t g_read_streams[OS_FDTD_MAX_DEVICES] = {};
cudaEvent_t g_read_ready[OS_FDTD_MAX_DEVICES] = {};

// Whether the pages of [p, p + bytes) are there (a sample of them; unknown counts as no).
bool resident(const void *p, size_t bytes) {
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), first = (uintptr_t)p;
    for (int k = 0; k < 16; ++k) {
        unsigned char in = 0;
        const uintptr_t at = (first + (bytes - 1) / 15 * k) & ~(page - 1);
        if (mincore((void *)at, page, &in) != 0 || !(in & 1)) return false;
    }
    return true;
}

bool pageable(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// The device's reader stream, behind the work queued on `stream` so far.
cudaError_t read_stream(int device, cudaStream_t stream, cudaStream_t *out) {
    cudaStream_t &s = g_read_streams[device];
    cudaEvent_t &ready = g_read_ready[device];
    cudaError_t err = s ? cudaSuccess : cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    if (err == cudaSuccess && !ready) err = cudaEventCreateWithFlags(&ready, cudaEventDisableTiming);
    if (err == cudaSuccess) err = cudaEventRecord(ready, stream);
    if (err == cudaSuccess) err = cudaStreamWaitEvent(s, ready, 0);
    *out = s;
    return err;
}

cudaError_t read_chunks(unsigned char *dst, const unsigned char *src, size_t bytes, int device, cudaStream_t stream,
                        unsigned char *slots, std::atomic<size_t> &next) {
    cudaError_t err = cudaSetDevice(device);
    cudaEvent_t done[2] = {nullptr, nullptr};
    for (auto &e : done)
        if (err == cudaSuccess) err = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    size_t at[2] = {bytes, bytes};   // chunk in flight per slot (bytes: none)
    for (int k = 0; err == cudaSuccess; k ^= 1) {
        const size_t begin = next.fetch_add(kReadChunk);
        if (begin < bytes) {
            const size_t n = bytes - begin < kReadChunk ? bytes - begin : kReadChunk;
            err = cudaMemcpyAsync(slots + k * kReadChunk, src + begin, n, cudaMemcpyDeviceToHost, stream);
            if (err == cudaSuccess) err = cudaEventRecord(done[k], stream);
            if (err != cudaSuccess) break;
            at[k] = begin;
        }
        if (at[k ^ 1] < bytes) {
            const size_t n = bytes - at[k ^ 1] < kReadChunk ? bytes - at[k ^ 1] : kReadChunk;
            err = cudaEventSynchronize(done[k ^ 1]);
            if (err == cudaSuccess) memcpy(dst + at[k ^ 1], slots + (k ^ 1) * kReadChunk, n);
            at[k ^ 1] = bytes;
        }
        if (at[0] >= bytes && at[1] >= bytes) break;
    }
    for (cudaEvent_t e : done)
        if (e) {
            cudaEventSynchronize(e);   // nothing may still write this thread's slots
            cudaEventDestroy(e);
        }
    return err;
}
}  // namespace

int read_back(void *dst, const void *src, size_t bytes, cudaStream_t stream) {
    std::unique_lock<std::mutex> lock(g_read_mutex, std::defer_lock);
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    int device = -1;
    if (bytes >= kReadMin && pageable(dst) && (bytes >= kReadMinResident || !resident(dst, bytes))) {
        // a capturing stream keeps the plain copy, and its error
        OS_CUDA(cudaGetDevice(&device));
        OS_CUDA(cudaStreamIsCapturing(stream, &capture));
    }
    if (device >= 0 && device < OS_FDTD_MAX_DEVICES && capture == cudaStreamCaptureStatusNone && lock.try_lock()) {
        if (!g_read_slots &&
            cudaHostAlloc((void **)&g_read_slots, kReadThreads * 2 * kReadChunk, cudaHostAllocPortable) != cudaSuccess) {
            g_read_slots = nullptr;
            cudaGetLastError();
        }
        if (g_read_slots) {
            cudaStream_t reader = nullptr;
            OS_CUDA(read_stream(device, stream, &reader));
            std::atomic<size_t> next{0};
            cudaError_t err[kReadThreads];
            std::vector<std::thread> threads;
            int started = 0;
            auto work = [&](int k) {
                err[k] = read_chunks(static_cast<unsigned char *>(dst), static_cast<const unsigned char *>(src), bytes,
                                     device, reader, g_read_slots + k * 2 * kReadChunk, next);
            };
            try {
                threads.reserve(kReadThreads - 1);
                for (; started < kReadThreads - 1; ++started) threads.emplace_back(work, started);
            } catch (...) {   // no more threads: those started and this one do the work
            }
            work(started);
            for (auto &t : threads) t.join();
            for (int k = 0; k <= started; ++k) OS_CUDA(err[k]);
            return OS_OK;
        }
    }
    OS_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream));
    OS_CUDA(cudaStreamSynchronize(stream));
    return OS_OK;
}

int pool_trim() {
    {
        std::lock_guard<std::mutex> lock(g_read_mutex);
        if (g_read_slots) cudaFreeHost(g_read_slots);
        g_read_slots = nullptr;
        for (cudaStream_t &s : g_read_streams) {
            if (s) cudaStreamDestroy(s);
            s = nullptr;
        }
        for (cudaEvent_t &e : g_read_ready) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
    }
    std::vector<PoolBlock> blocks;
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        for (auto &kv : g_pool)
            for (auto &b : kv.second) blocks.push_back(b);
        g_pool.clear();
        g_pool_bytes = 0;
    }
    for (auto &b : blocks) {
        if (b.events)
            for (cudaEvent_t ev : b.events->events) cudaEventSynchronize(ev);
        cudaFree(b.ptr);
    }
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    for (auto &b : blocks) unref(b.events);
    return OS_OK;
}

}  // namespace os

extern "C" int os_fdtd_pool_trim(void) { return os::pool_trim(); }

extern "C" int os_fdtd_last_error(char *buf, size_t n) {
    const std::string &msg = os::last_error();
    if (buf && n) {
        size_t len = msg.size() < n - 1 ? msg.size() : n - 1;
        memcpy(buf, msg.data(), len);
        buf[len] = '\0';
    }
    return (int)msg.size();
}

// GaussianPulse.__call__ for a float time, in double with the C library's functions, which Python's math module calls
// too (core/sources.py:40-46): exp(-((t - t0) / tau) ** 2) sin(2 pi f0 (t - t0)).
extern "C" int os_gaussian_values(double f0, double tau, double t0, const double *t, int64_t n, double *out) {
    OS_CHECK(n >= 0 && (n == 0 || (t && out)), OS_ERR_INVALID, "os_gaussian_values: null argument");
    volatile double two = 2.0;   // pow as Python's ** calls it, not folded to a product
    for (int64_t k = 0; k < n; ++k) {
        const double delay = t[k] - t0;
        out[k] = std::exp(-std::pow(delay / tau, two)) * std::sin(2.0 * 3.141592653589793 * f0 * delay);
    }
    return OS_OK;
}

extern "C" int os_fdtd_version(void) { return 100; }

extern "C" int os_fdtd_host_alloc(size_t bytes, void **out) {
    OS_CHECK(out, OS_ERR_INVALID, "os_fdtd_host_alloc: null argument");
    *out = nullptr;
    if (bytes == 0) return OS_OK;
    OS_CUDA(cudaHostAlloc(out, bytes, cudaHostAllocPortable));
    return OS_OK;
}

extern "C" int os_fdtd_host_free(void *ptr) {
    if (ptr) OS_CUDA(cudaFreeHost(ptr));
    return OS_OK;
}
