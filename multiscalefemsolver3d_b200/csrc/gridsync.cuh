// Grid-wide barrier and deterministic reductions for cooperative kernels (one launch, every CTA
// resident): the persistent Krylov loops.
//
// A barrier is one atomic arrival per CTA on a counter that only grows, and a poll of it by one
// thread.  Every wait is bounded: a CTA whose wait expires raises `abort` and leaves the kernel, the
// others see the flag or expire as well, and the host reports it.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace msfem {

struct GridBar {
    unsigned int arrived;
    unsigned int abort;
};

constexpr int kGridSpins = 1 << 22;

__device__ __forceinline__ unsigned int load_acquire(const unsigned int* p)
{
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// One CTA's view of the barrier: construct once per kernel with a shared int.
struct GridSync {
    GridBar* bar;
    unsigned int target = 0;
    int* ok;  // shared
    __device__ GridSync(GridBar* b, int* shared_ok) : bar(b), ok(shared_ok) {}
    // global writes of every CTA before it are visible to every CTA after it; false: give up
    __device__ __forceinline__ bool sync()
    {
        target += gridDim.x;
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(&bar->arrived), "r"(1u) : "memory");
            int good = 1;
            for (int spin = 0; (int)(load_acquire(&bar->arrived) - target) < 0; spin++)
                if (spin >= kGridSpins || ((spin & 1023) == 1023 && load_acquire(&bar->abort))) {
                    atomicExch(&bar->abort, 1u);
                    good = 0;
                    break;
                }
            *ok = good;
        }
        __syncthreads();
        return *ok != 0;
    }
};

// coherent load of a vector that the running kernel also writes (never the read-only path)
template <class T>
__device__ __forceinline__ T load_shared_vector(const T* p);
template <>
__device__ __forceinline__ float load_shared_vector<float>(const float* p)
{
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
template <>
__device__ __forceinline__ double load_shared_vector<double>(const double* p)
{
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

}  // namespace msfem
