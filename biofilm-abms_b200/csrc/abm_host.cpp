// Device-to-host copies into pageable memory, by several host threads.
//
// A frame goes to memory that the caller has just allocated: the copy's time is page faults
// and one core's memcpy out of the driver's staging buffer (4.5 GB/s: 7.8 ms for the 35 MB of
// 200,000 cells, a quarter of the 200 steps before it), not the bus.  Here each of up to
// eight threads takes pieces of the range, brings a piece into pinned memory of its own and
// copies it out, so that the faults and the copying run side by side.  The pinned pieces and
// their streams are shared by the contexts of the process: made at the first large copy,
// given back when the last context is destroyed.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <exception>
#include <thread>
#include <vector>
#include <cuda_runtime.h>
#include "abm_host.hpp"

namespace abm {

namespace {

const size_t PIECE = 512 << 10;
const int MAX_WORKERS = 8;
// Below this a single copy is faster: starting and joining the threads takes 0.2-0.3 ms (forces
// of 50,021 cells, 2.4 MB: 0.66 ms alone, 0.95 with threads; 5.3 MB: 5.9 and 6.3; 17.6 MB: 12.3
// and 11.5; 35 MB: 29.6 and 24.2, each with the steps before the copy).
const size_t MIN_BYTES = 12 << 20;

struct Worker {
    void* pinned = nullptr;
    cudaStream_t st = nullptr;
    int dev = -1;
};

std::mutex g_mu;                 // held by the copy that uses the workers
Worker g_workers[MAX_WORKERS];
std::mutex g_users_mu;
int g_users = 0;

void drop(Worker& w)
{
    if (w.st) cudaStreamDestroy(w.st);
    if (w.pinned) cudaFreeHost(w.pinned);
    w = Worker();
}

// a worker's pinned piece and stream on `dev`; false if they cannot be had
bool ready(Worker& w, int dev)
{
    if (w.pinned && w.dev == dev) return true;
    drop(w);
    w.dev = dev;
    if (cudaHostAlloc(&w.pinned, PIECE, cudaHostAllocPortable) == cudaSuccess &&
        cudaStreamCreateWithFlags(&w.st, cudaStreamNonBlocking) == cudaSuccess)
        return true;
    cudaGetLastError();
    drop(w);
    return false;
}

struct Piece {
    char* dst;
    const char* src;
    size_t bytes;
};

}   // namespace

void host_copy_retain()
{
    std::lock_guard<std::mutex> l(g_users_mu);
    ++g_users;
}

void host_copy_release()
{
    std::lock_guard<std::mutex> l(g_users_mu);
    if (--g_users > 0) return;
    std::lock_guard<std::mutex> copy(g_mu);
    for (Worker& w : g_workers) drop(w);
}

cudaError_t copy_to_host(int dev, void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
                         size_t height, cudaStream_t st)
{
    if (width == 0 || height == 0) return cudaSuccess;
    const size_t total = width * height;
    auto plain = [&]() {
        cudaError_t e = cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, height, cudaMemcpyDeviceToHost, st);
        return e != cudaSuccess ? e : cudaStreamSynchronize(st);
    };
    if (total < MIN_BYTES) return plain();
    // pinned and managed destinations take the copy as it is
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) { cudaGetLastError(); return plain(); }
    if (at.type != cudaMemoryTypeUnregistered) return plain();
    // another copy has the workers: no waiting for it
    std::unique_lock<std::mutex> lock(g_mu, std::try_to_lock);
    if (!lock.owns_lock()) return plain();
    try
    {
        std::vector<Piece> pieces;
        const bool whole = dpitch == width && spitch == width;
        const size_t rows = whole ? 1 : height, len = whole ? total : width;
        for (size_t r = 0; r < rows; ++r)
            for (size_t o = 0; o < len; o += PIECE)
                pieces.push_back({static_cast<char*>(dst) + r * dpitch + o, static_cast<const char*>(src) + r * spitch + o,
                                  std::min(PIECE, len - o)});
        const int cores = std::max(1u, std::thread::hardware_concurrency());
        const int want = (int)std::min<size_t>({pieces.size(), (size_t)MAX_WORKERS, (size_t)std::max(1, cores / 2)});
        int workers = 0;
        while (workers < want && ready(g_workers[workers], dev)) ++workers;
        if (workers < 2) return plain();
        // what the stream still has to write
        cudaError_t e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        std::atomic<size_t> next{0};
        std::atomic<int> failed{(int)cudaSuccess};
        auto work = [&](int k) {
            Worker& w = g_workers[k];
            if (cudaSetDevice(dev) != cudaSuccess) { failed = (int)cudaErrorInvalidDevice; return; }
            for (size_t q; failed == (int)cudaSuccess && (q = next++) < pieces.size();)
            {
                const Piece& p = pieces[q];
                cudaError_t c = cudaMemcpyAsync(w.pinned, p.src, p.bytes, cudaMemcpyDeviceToHost, w.st);
                if (c == cudaSuccess) c = cudaStreamSynchronize(w.st);
                if (c != cudaSuccess) { failed = (int)c; return; }
                memcpy(p.dst, w.pinned, p.bytes);
            }
        };
        std::vector<std::thread> threads;
        threads.reserve(workers);
        // a thread that cannot be started (no thread, or no memory for one) leaves its pieces to
        // the others; the ones that run are joined in any case
        try { for (int k = 1; k < workers; ++k) threads.emplace_back(work, k); }
        catch (const std::exception&) {}
        work(0);
        for (std::thread& t : threads) t.join();
        return (cudaError_t)failed.load();
    }
    catch (const std::bad_alloc&)
    {
        return plain();
    }
}

}   // namespace abm
