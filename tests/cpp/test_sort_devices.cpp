// The radix sorts on two devices of one process, over a stand-in for the CUDA runtime: a launch
// that takes more dynamic shared memory than 48 KB is refused, as the runtime refuses it, where
// the kernel was not opted in on the current device. No GPU is used and no kernel runs.
#include <cstdio>
#include <map>
#include <set>
#include <utility>

#include "sort.cuh"

namespace
{
    int g_device = 0;
    std::map<std::pair<int, const void*>, int> g_limit;     // (device, kernel) -> opted-in bytes
    int g_refused = 0, g_made = 0;
}

extern "C"
{
    void** __cudaRegisterFatBinary(void*) { static void* h = nullptr; return &h; }
    void __cudaRegisterFatBinaryEnd(void**) {}
    void __cudaUnregisterFatBinary(void**) {}
    void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
    void __cudaInitModule(void**) {}
    unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
    cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
    cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
    cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorUnknown; }
    cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorUnknown; }
    cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
    cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 4; return cudaSuccess; }
    cudaError_t cudaGetLastError(void) { return cudaSuccess; }
    cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
    {
        *n = 3;
        return cudaSuccess;
    }
    cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t)
    {
        *n = 3;
        return cudaSuccess;
    }
    cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int bytes)
    {
        g_limit[{ g_device, f }] = bytes;
        return cudaSuccess;
    }
    cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**)
    {
        const auto it = g_limit.find({ g_device, f });
        const bool ok = c->dynamicSmemBytes <= 48 * 1024
                        || (it != g_limit.end() && static_cast<size_t>(it->second) >= c->dynamicSmemBytes);
        ++(ok ? g_made : g_refused);
        return ok ? cudaSuccess : cudaErrorInvalidValue;
    }
}

int main()
{
    for (g_device = 0; g_device < 2; ++g_device)
        for (const size_t n : { size_t(3000), size_t(1) << 20 })     // both forms of a pass
        {
            nbg::SortSetup setup;       // a context's own
            uint64_t launches = 0, keys[2] = {}, temp = 0;
            uint32_t vals[2] = {};
            bool alt = false;
            unsigned err = 0, run = 0;
            if (nbg::setup_sort(&setup) != cudaSuccess)
                return 2;
            const cudaError_t a = nbg::radix_sort_pairs(keys, vals, keys + 1, vals + 1, n, 18, 63, &temp, nullptr,
                                                        &launches, &alt, &err, false, setup);
            const cudaError_t b = nbg::radix_sort_if(keys, vals, keys + 1, vals + 1, n, 0, 63, &temp, 5, nullptr,
                                                     &launches, &err, &run, setup);
            std::printf("device %d, %zu keys: %d %d, %d launches made, %d refused\n", g_device, n, a, b, g_made, g_refused);
            if (a != cudaSuccess || b != cudaSuccess || g_refused)
                return 1;
        }
    return 0;
}
