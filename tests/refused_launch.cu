// A build launch with more blocks than the device holds at once: the runtime refuses it, the
// launch wrapper hands the refusal on, and nothing runs.  Linked against libabm_b200.so.
#include <cstdio>
#include <cstring>
#include "abm_kernels.cuh"

using namespace abm;

int main()
{
    Ctrl h;
    memset(&h, 0, sizeof(h));
    Ctrl* ctrl = nullptr;
    if (cudaMalloc(&ctrl, sizeof(Ctrl)) != cudaSuccess) return 2;
    if (cudaMemcpy(ctrl, &h, sizeof(Ctrl), cudaMemcpyHostToDevice) != cudaSuccess) return 2;
    BuildArgs a{};
    a.ctrl = ctrl;
    LaunchShape shape;
    shape.blocks = 1 << 20;
    const cudaError_t e = launch_build(a, BUILD_RECORDS, shape, 0);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    if (cudaMemcpy(&h, ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("%s %d %d\n", cudaGetErrorName(e), h.status, h.halted);
    return 0;
}
