// copy_to_host against stand-ins of the CUDA calls it makes, with memory running out at each of
// its allocations in turn: the data must arrive and the process must go on.  Prints "ok".
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>
#include "abm_host.hpp"

static std::atomic<int> g_left{-1};             // allocations until one fails; negative: none does

void* operator new(std::size_t n)
{
    if (g_left >= 0 && g_left-- == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

extern "C" {
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t)
{
    for (size_t r = 0; r < h; ++r) std::memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*)
{
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return (*p = std::malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)1; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
}

int main()
{
    const size_t rows = 5, width = (3 << 20) + 24, pitch = width + 40;      // 15 MB: past the threshold
    std::vector<unsigned char> src(rows * width), dst(rows * pitch);
    for (size_t i = 0; i < src.size(); ++i) src[i] = (unsigned char)(i * 2654435761u >> 13);
    abm::host_copy_retain();
    int failed = 0;
    for (int k = -1; k < 64; ++k)
    {
        std::memset(dst.data(), 0xee, dst.size());
        g_left = k;
        const cudaError_t e = abm::copy_to_host(0, dst.data(), pitch, src.data(), width, width, rows, nullptr);
        failed += k >= 0 && g_left < 0;
        g_left = -1;
        if (e != cudaSuccess) { std::printf("allocation %d: error %d\n", k, (int)e); return 1; }
        for (size_t r = 0; r < rows; ++r)
            if (std::memcmp(dst.data() + r * pitch, src.data() + r * width, width)) { std::printf("allocation %d: row %zu\n", k, r); return 1; }
    }
    abm::host_copy_release();
    if (failed < 3) { std::printf("only %d allocations failed\n", failed); return 1; }
    std::printf("ok\n");
    return 0;
}
