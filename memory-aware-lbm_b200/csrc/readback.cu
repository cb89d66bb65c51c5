// readback.cu -- results into the caller's arrays through pinned memory.
//
// A copy of a large result straight into a fresh pageable array runs at about 5 GB/s: one thread of the
// driver copies through its own staging buffer and takes every page fault of the array (1.6 GB of a 16384 x
// 4096 channel's fields: 333 ms).  Here the kernels write each chunk into pinned memory over the link (no
// device buffer), and several threads, each with two chunks of its own so that one fills while the other is
// copied, move them into the array and share its page faults.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <exception>
#include <thread>
#include "readback.h"

namespace lbgpu {

namespace {

constexpr size_t kChunk = (size_t)1 << 20;         // bytes of a chunk
constexpr int kThreads = 8;

// Pinned memory between calls: one buffer (the size that the largest call took, at most 64 MiB or two rows or
// columns), given back with the last lattice.
std::mutex g_mu;
void *g_spare = nullptr;
size_t g_spare_bytes = 0;

cudaError_t take_pinned(size_t bytes, void **p, size_t *got)
{
    void *old = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (g_spare && g_spare_bytes >= bytes) {
            *p = g_spare;
            *got = g_spare_bytes;
            g_spare = nullptr;
            return cudaSuccess;
        }
        old = g_spare;
        g_spare = nullptr;
    }
    if (old) cudaFreeHost(old);
    *got = bytes;
    return cudaHostAlloc(p, bytes, cudaHostAllocPortable | cudaHostAllocMapped);
}

void give_pinned(void *p, size_t bytes)
{
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (!g_spare) {
            g_spare = p;
            g_spare_bytes = bytes;
            return;
        }
    }
    cudaFreeHost(p);
}

}  // namespace

void read_back_release()
{
    void *p = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        p = g_spare;
        g_spare = nullptr;
    }
    if (p) cudaFreeHost(p);
}

cudaError_t read_back(int device, cudaStream_t stream, long long items, size_t item_bytes, RangeFn<double> fill,
                      RangeFn<const double> take)
{
    if (items <= 0 || item_bytes == 0) return cudaStreamSynchronize(stream);
    int before = device;
    if (cudaError_t e = cudaGetDevice(&before)) return e;
    const size_t total = (size_t)items * item_bytes;
    const long long per = std::max<long long>(1, (long long)(std::min(kChunk, (total + 3) / 4) / item_bytes));
    const size_t slot = ((size_t)per * item_bytes + 255) / 256 * 256;
    const int cores = std::max(1, (int)std::thread::hardware_concurrency() / 2);
    // one thread for every 4 MiB (more threads only contend for page faults: 6 MB 1.1 ms on 6 threads, 0.6 on one), and no more than 64 MiB of chunks
    int want = (int)std::min<size_t>((size_t)std::min(kThreads, cores), std::max<size_t>(1, total >> 22));
    want = (int)std::max<size_t>(1, std::min<size_t>((size_t)want, ((size_t)64 << 20) / (2 * slot)));
    void *mem = nullptr;
    size_t bytes = 0;
    if (cudaError_t e = take_pinned(2 * slot * (size_t)want, &mem, &bytes)) return e;
    std::atomic<long long> next(0);
    std::atomic<int> failed(0);
    cudaError_t errors[kThreads] = {};
    auto work = [&](int t) {
        double *buf[2];
        cudaEvent_t ev[2] = {nullptr, nullptr};
        long long k0[2] = {-1, -1};
        cudaError_t e = cudaSetDevice(device);
        for (int b = 0; b < 2; ++b) {
            buf[b] = reinterpret_cast<double *>(static_cast<char *>(mem) + (size_t)(2 * t + b) * slot);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev[b], cudaEventDisableTiming);
        }
        auto start = [&](int b) {
            k0[b] = -1;
            if (e != cudaSuccess || failed.load()) return;
            const long long k = next.fetch_add(per);
            if (k >= items) return;
            fill(k, std::min(items, k + per), buf[b]);
            e = cudaGetLastError();
            if (e == cudaSuccess) e = cudaEventRecord(ev[b], stream);
            if (e == cudaSuccess) k0[b] = k;
        };
        start(0);
        for (int b = 0; k0[b] >= 0; b ^= 1) {
            start(b ^ 1);
            const cudaError_t w = cudaEventSynchronize(ev[b]);
            if (w != cudaSuccess) {
                e = w;
                break;
            }
            take(k0[b], std::min(items, k0[b] + per), buf[b]);
        }
        for (int b = 0; b < 2; ++b)
            if (ev[b]) cudaEventDestroy(ev[b]);
        if (e != cudaSuccess) failed.store(1);
        errors[t] = e;
    };
    std::thread team[kThreads];
    for (int t = 1; t < want; ++t) {
        try {
            team[t] = std::thread(work, t);
        } catch (const std::exception &) {
            break;                       // fewer threads: the others take their chunks
        }
    }
    work(0);
    for (std::thread &t : team)
        if (t.joinable()) t.join();
    cudaError_t first = cudaSuccess;
    for (cudaError_t e : errors)
        if (first == cudaSuccess) first = e;
    if (first != cudaSuccess) cudaStreamSynchronize(stream);   // chunks in flight write the pinned memory
    give_pinned(mem, bytes);
    if (before != device) cudaSetDevice(before);
    return first;
}

}  // namespace lbgpu
