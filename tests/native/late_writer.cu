// A kernel that lets its dependents start at once and writes long after: what a kernel ahead of ours may do at worst.
#include <cuda_runtime.h>

#include <algorithm>

namespace {
constexpr int kThreads = 256;

__global__ void __launch_bounds__(kThreads) late_copy(uint4* dst, const uint4* src, size_t n, long long cycles)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long begin = clock64();
    while (clock64() - begin < cycles) __nanosleep(200);
    for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (size_t)gridDim.x * kThreads) dst[i] = src[i];
}
}  // namespace

// `blocks` of them leave most of the device to the kernel behind
extern "C" int late_copy_launch(void* dst, const void* src, size_t bytes, int blocks, int cycles, void* stream)
{
    if (bytes % 16 || blocks <= 0) return -1;
    late_copy<<<blocks, kThreads, 0, (cudaStream_t)stream>>>((uint4*)dst, (const uint4*)src, bytes / 16, std::min(cycles, 2000000));
    return (int)cudaGetLastError();
}
