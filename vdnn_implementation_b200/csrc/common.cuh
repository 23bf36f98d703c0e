// Shared helpers for the sm_100a kernels: status plumbing, launch sizing, fast integer division.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "once.h"
#include "vdnn_b200.h"

namespace vdnn {

// Last failing runtime call of this thread, reported by vdnn_last_cuda_error().
extern thread_local int g_last_cuda_error;
// Launch counter (all kernels of this library), reported through vdnn_network_stats.
extern unsigned long long g_kernel_launches;

inline int cuda_fail(cudaError_t e) {
    g_last_cuda_error = static_cast<int>(e);
    (void)cudaGetLastError();
    return VDNN_ERR_CUDA;
}

#define VDNN_CUDA(call)                                              \
    do {                                                             \
        cudaError_t _e = (call);                                     \
        if (_e != cudaSuccess) return ::vdnn::cuda_fail(_e);         \
    } while (0)

// After a <<<>>> launch: count it and surface launch-configuration errors.
#define VDNN_LAUNCHED()                                              \
    do {                                                             \
        ++::vdnn::g_kernel_launches;                                 \
        cudaError_t _e = cudaPeekAtLastError();                      \
        if (_e != cudaSuccess) return ::vdnn::cuda_fail(_e);         \
    } while (0)

// B200 has 148 SMs; grids of the bandwidth kernels are sized in whole multiples of the SM count
// (queried once per device) so that every SM gets the same number of resident blocks.
int sm_count();

// Raises a kernel's limit of dynamic shared memory, once per device and kernel (each instance of a template is a place of its
// own); no thread launches before it is raised.
#define VDNN_ALLOW_SHARED(dev, kern, bytes)                                                                            \
    do {                                                                                                               \
        static ::vdnn::OncePerDevice _once;                                                                            \
        VDNN_CUDA(_once.run((dev), [&]() { return cudaFuncSetAttribute((kern), cudaFuncAttributeMaxDynamicSharedMemorySize, (bytes)); })); \
    } while (0)

inline cudaStream_t as_stream(void* s) { return static_cast<cudaStream_t>(s); }

template <typename T>
__host__ __device__ constexpr T ceil_div(T a, T b) { return (a + b - 1) / b; }

// Division by a run-time constant with one mul.hi (valid for dividends below 2^31).
struct FastDiv {
    uint32_t d, mul, shr;
    FastDiv() : d(1), mul(0), shr(0) {}
    explicit FastDiv(uint32_t denom) : d(denom), mul(0), shr(0) {
        if (denom > 1) {
            uint32_t lg = 0;
            while ((1u << lg) < denom) ++lg;
            const uint32_t p = 31 + lg;
            mul = static_cast<uint32_t>(((1ull << p) + denom - 1) / denom);
            shr = p - 32;
        }
    }
    __host__ __device__ __forceinline__ uint32_t div(uint32_t n) const {
#ifdef __CUDA_ARCH__
        return d == 1 ? n : (__umulhi(n, mul) >> shr);
#else
        return n / d;
#endif
    }
    __host__ __device__ __forceinline__ void divmod(uint32_t n, uint32_t& q, uint32_t& r) const {
        q = div(n);
        r = n - q * d;
    }
};

namespace tc {

// The kernels of one call, or of a step's last layers, follow each other within microseconds of work.  Launched like this a
// kernel may start while its predecessor in the stream still runs (which says so by follow_up()) and sets itself up; its
// after_predecessor(), before the first global access, waits until all of the predecessor's results are visible.  A kernel
// launched otherwise waits as always.
// Measured: 5 x 48 x 27 x 31 -> 80, 3 x 3, forward and backward (nine kernels, 64 us of work): 78 -> 65 us.
__device__ __forceinline__ void after_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void follow_up() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class Kernel, class... Args>
inline cudaError_t launch_early(Kernel kern, dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cfg.attrs = attr; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace tc

}  // namespace vdnn
