// A barrier whose wait runs out, and what follows on the same control record.  One block waits
// for a second that is never launched: the wait is bounded, so the kernel ends by itself with
// an error status.  Then the launches that would use what the barrier guards must leave at once
// and change nothing.  Linked against libabm_b200.so; prints "ok" and returns 0.
#include <cstdio>
#include <cstring>
#include <vector>
#include "abm_grid.cuh"

using namespace abm;

#define CK(call) do { cudaError_t e_ = (call); if (e_ != cudaSuccess) { \
    printf("%s: %s\n", #call, cudaGetErrorString(e_)); return 2; } } while (0)
#define EXPECT(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

__global__ void wait_for_two(GridBar* bar, Ctrl* ctrl, int* passed)
{
    const bool ok = grid_barrier(bar, 2, ctrl);
    if (threadIdx.x == 0) *passed = ok;
}

// n elements of T, every byte 0x5a
template <class T> T* marked(size_t n)
{
    void* p = nullptr;
    if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess || cudaMemset(p, 0x5a, n * sizeof(T)) != cudaSuccess) return nullptr;
    return static_cast<T*>(p);
}
template <class T> bool untouched(const T* p, size_t n)
{
    std::vector<unsigned char> h(n * sizeof(T));
    if (cudaMemcpy(h.data(), p, h.size(), cudaMemcpyDeviceToHost) != cudaSuccess) return false;
    for (unsigned char b : h) if (b != 0x5a) return false;
    return true;
}

int main()
{
    const int n = 64, cap_nbr = 8, bins = 1 << 12;
    Ctrl h;
    memset(&h, 0, sizeof(h));
    h.n = n;
    Ctrl* ctrl;
    GridBar* bar;
    int* passed;
    CK(cudaMalloc(&ctrl, sizeof(Ctrl)));
    CK(cudaMemcpy(ctrl, &h, sizeof(Ctrl), cudaMemcpyHostToDevice));
    CK(cudaMalloc(&bar, sizeof(GridBar)));
    CK(cudaMemset(bar, 0, sizeof(GridBar)));
    CK(cudaMalloc(&passed, sizeof(int)));
    CK(cudaMemset(passed, 0xff, sizeof(int)));
    wait_for_two<<<1, 64>>>(bar, ctrl, passed);
    CK(cudaGetLastError());
    CK(cudaDeviceSynchronize());
    int ok = -1;
    CK(cudaMemcpy(&ok, passed, sizeof(int), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(&h, ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost));
    EXPECT(ok == 0);
    EXPECT(h.status == ST_BARRIER);
    EXPECT(h.halted == HALT_LOST);

    // a rebuild, as a cluster and as a cooperative grid
    Geom* geom = marked<Geom>(n);
    CK(cudaMemset(geom, 0, n * sizeof(Geom)));
    BuildArgs a{};
    a.geom = geom; a.vel = marked<Vel>(n); a.phys = marked<Phys>(n); a.ctrl = ctrl; a.bar = bar;
    a.bbox = marked<int>(8 * 16); a.part = marked<int2>(16);
    a.bin_count = marked<int>(bins); a.bin_start = marked<int>(2 * bins);
    a.key = marked<int>(n); a.slot = marked<int>(n); a.sorted_cell = marked<int>(n); a.sorted_key = marked<int>(n);
    a.sorted_pos = marked<float4>(n); a.sorted_dir = marked<float4>(n);
    a.cap_bins = bins; a.cap_cells = n;
    a.bp = {3.6, 10.8, cap_nbr};
    a.scratch = marked<int>(n * cap_nbr); a.count = marked<int>(n); a.row_ptr = marked<int>(n + 1);
    a.col = marked<int>(n * cap_nbr); a.lower_end = marked<int>(n); a.pairs = marked<int4>(n * cap_nbr / 2 + 1);
    for (int cluster = 0; cluster < 2; ++cluster)
    {
        LaunchShape s;
        s.blocks = 2;
        s.cluster = cluster;
        launch_build(a, BUILD_NEIGHBORS, s, 0);
        CK(cudaGetLastError());
    }
    // a pair pass and the row sums of the forces call
    ForceParams fp;
    memset(&fp, 0, sizeof(fp));
    fp.R = 0.8;
    double4* jbuf = marked<double4>(n * cap_nbr);
    Gen6* fcc = marked<Gen6>(n);
    ActiveList al{};
    al.act = marked<int4>(n * cap_nbr / 2 + 1); al.n_act = marked<int>(n); al.keep = marked<unsigned char>(n * cap_nbr);
    al.gref = marked<Geom>(n); al.row_ptr = a.row_ptr; al.bar = bar;
    launch_pair_screened(geom, ctrl, fp, nullptr, nullptr, fcc, jbuf, 0, n * cap_nbr, n, 148, 0, 1, 3, 0, 0, a.pairs,
                         marked<int>(n * cap_nbr / 2 + 1), al, n, 1);
    CK(cudaGetLastError());
    CK(cudaDeviceSynchronize());
    EXPECT(untouched(a.bin_count, bins) && untouched(a.bin_start, 2 * bins) && untouched(a.row_ptr, n + 1));
    EXPECT(untouched(a.col, n * cap_nbr) && untouched(a.pairs, n * cap_nbr / 2 + 1) && untouched(a.sorted_cell, n));
    EXPECT(untouched(jbuf, n * cap_nbr) && untouched(al.act, n * cap_nbr / 2 + 1) && untouched(al.n_act, n));
    std::vector<Gen6> f(n);
    CK(cudaMemcpy(f.data(), fcc, n * sizeof(Gen6), cudaMemcpyDeviceToHost));
    for (const Gen6& g : f) for (double x : g.f) EXPECT(x != x);
    GridBar rec;
    CK(cudaMemcpy(&rec, bar, sizeof(rec), cudaMemcpyDeviceToHost));
    EXPECT(rec.count == 1 && rec.gen == 0);                 // nobody waited on it again
    CK(cudaMemcpy(&h, ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost));
    EXPECT(h.status == ST_BARRIER && h.halted == HALT_LOST && h.rebuilds == 0);
    printf("ok\n");
    return 0;
}
