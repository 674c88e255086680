// Copies between the caller's pageable arrays and the device.
//
// A pageable cudaMemcpy runs one host copy through the driver's own pinned
// buffer: 33 MB take 3.1 ms to the device and 2.4 ms back (13 ms where the
// destination has no pages yet), of which the link needs 0.6.  Here a few
// threads move chunks through a pinned buffer of 8 MB, two chunks each, so
// that host copies run side by side and under the transfers.  A solve from
// 96 x 128 x 112 host arrays (45 MB in, 33 MB out) 15.1 -> 11.5 ms, the map of
// its result 5.1 -> 3.3; below 4 MB the two ways take the same time (56^3 map
// 1.7 ms).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include <sys/mman.h>
#include <unistd.h>

#include "dt_internal.h"

namespace dtb {
namespace {

constexpr size_t CHUNK = size_t(1) << 20;
constexpr int WORKERS = 4, SLOTS = 2;  // chunks in flight per worker

std::mutex g_staging_mutex;  // held for a whole copy
char *g_staging = nullptr;   // WORKERS * SLOTS chunks, pinned, for every device

bool pageable(const void *p) {
    cudaPointerAttributes a = {};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

struct Copy {
    char *host;
    char *device;
    size_t bytes;
    bool in;  // host to device
    cudaStream_t stream;
    cudaEvent_t events[WORKERS * SLOTS];
    std::atomic<size_t> next{0};
    std::atomic<int> error{cudaSuccess};

    void fail(cudaError_t e) {
        int none = cudaSuccess;
        if (e != cudaSuccess) error.compare_exchange_strong(none, (int) e);
    }
    // The next chunk's offset, or `bytes` when none is left.
    size_t take() { return error.load() == cudaSuccess ? std::min(next.fetch_add(CHUNK), bytes) : bytes; }
    size_t length(size_t at) const { return std::min(CHUNK, bytes - at); }

    void work(int worker) {
        char *slot = g_staging + (size_t) worker * SLOTS * CHUNK;
        cudaEvent_t *done = events + worker * SLOTS;
        size_t at[SLOTS];  // chunk in each slot
        for (int k = 0; k < SLOTS; ++k) at[k] = bytes;
        auto finish = [&](int k) {  // waits for the slot's transfer and empties it
            if (at[k] == bytes) return;
            fail(cudaEventSynchronize(done[k]));
            if (!in && error.load() == cudaSuccess) std::memcpy(host + at[k], slot + k * CHUNK, length(at[k]));
            at[k] = bytes;
        };
        for (int k = 0;; k = (k + 1) % SLOTS) {
            finish(k);
            const size_t c = take();
            if (c == bytes) break;
            if (in) std::memcpy(slot + k * CHUNK, host + c, length(c));
            fail(in ? cudaMemcpyAsync(device + c, slot + k * CHUNK, length(c), cudaMemcpyHostToDevice, stream)
                    : cudaMemcpyAsync(slot + k * CHUNK, device + c, length(c), cudaMemcpyDeviceToHost, stream));
            fail(cudaEventRecord(done[k], stream));
            at[k] = c;
        }
        for (int k = 0; k < SLOTS; ++k) finish(k);
    }
};

// The staged copy, or false (nothing done) where a plain one serves.
bool staged(void *host, void *device, size_t bytes, bool in, cudaStream_t stream, cudaError_t *result) {
    if (bytes < HOST_COPY_STAGED || !pageable(host)) return false;
    std::unique_lock<std::mutex> lock(g_staging_mutex, std::try_to_lock);
    if (!lock.owns_lock()) return false;  // another thread's copy has the buffer
    if (!g_staging && cudaHostAlloc(&g_staging, WORKERS * SLOTS * CHUNK, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        g_staging = nullptr;
        return false;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    Copy c;
    c.host = static_cast<char *>(host);
    c.device = static_cast<char *>(device);
    c.bytes = bytes;
    c.in = in;
    c.stream = stream;
    int made = 0;
    while (made < WORKERS * SLOTS && cudaEventCreateWithFlags(&c.events[made], cudaEventDisableTiming) == cudaSuccess)
        ++made;
    const bool ok = made == WORKERS * SLOTS;
    if (ok) {
        std::vector<std::thread> helpers;
        try {
            helpers.reserve(WORKERS - 1);
            for (int w = 1; w < WORKERS; ++w)
                helpers.emplace_back([&c, w, dev] {
                    const cudaError_t e = cudaSetDevice(dev);
                    if (e == cudaSuccess) c.work(w);
                    else c.fail(e);
                });
        } catch (...) {  // fewer helpers: the chunks go to those there are
        }
        c.work(0);
        for (std::thread &t : helpers) t.join();
        *result = (cudaError_t) c.error.load();
        if (*result != cudaSuccess) cudaStreamSynchronize(stream);  // no transfer is left on the buffer
    } else {
        cudaGetLastError();
    }
    for (int i = 0; i < made; ++i) cudaEventDestroy(c.events[i]);
    return ok;
}

}  // namespace

cudaError_t copy_from_host(void *device, const void *host, size_t bytes, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    if (staged(const_cast<void *>(host), device, bytes, true, s, &e)) return e;
    return cudaMemcpyAsync(device, host, bytes, cudaMemcpyHostToDevice, s);
}

cudaError_t copy_to_host(void *host, const void *device, size_t bytes, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    if (staged(host, const_cast<void *>(device), bytes, false, s, &e)) return e;
    return cudaMemcpyAsync(host, device, bytes, cudaMemcpyDeviceToHost, s);
}

void release_host_staging() {
    std::lock_guard<std::mutex> lock(g_staging_mutex);
    if (g_staging) cudaFreeHost(g_staging);
    g_staging = nullptr;
}

ResultPages::~ResultPages() {
    for (std::thread &t : threads_) t.join();
}

void ResultPages::populate(void *array, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
    constexpr size_t MAX_THREADS = 4, PER_THREAD = size_t(16) << 20;
    if (bytes < HOST_COPY_STAGED) return;
    const uintptr_t page = (uintptr_t) sysconf(_SC_PAGESIZE);
    const uintptr_t lo = reinterpret_cast<uintptr_t>(array) / page * page;
    const uintptr_t hi = (reinterpret_cast<uintptr_t>(array) + bytes + page - 1) / page * page;
    const size_t n = std::min(bytes / PER_THREAD + 1, MAX_THREADS - std::min(MAX_THREADS, threads_.size()));
    if (n == 0) return;
    const uintptr_t part = ((hi - lo) / n + page - 1) / page * page;
    try {
        for (uintptr_t at = lo; at < hi; at += part)
            threads_.emplace_back([at, len = (size_t) std::min(part, hi - at)] {
                madvise(reinterpret_cast<void *>(at), len, MADV_POPULATE_WRITE);
            });
    } catch (...) {  // no thread to be had: the copy takes the faults
    }
#else
    (void) array;
    (void) bytes;
#endif
}

}  // namespace dtb
