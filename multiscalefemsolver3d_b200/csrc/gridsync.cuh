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
    // one thread's arrival (with the CTA's writes, after a CTA barrier) and wait for `target`
    __device__ __forceinline__ void arrive_and_wait()
    {
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
    // global writes of every CTA before it are visible to every CTA after it; false: give up
    __device__ __forceinline__ bool sync()
    {
        target += gridDim.x;
        __syncthreads();
        if (threadIdx.x == 0) arrive_and_wait();
        __syncthreads();
        return *ok != 0;
    }
};

// Sums of a few values over the grid, an ordered barrier at the same time: a CTA's part goes to global
// memory ahead of its arrival, and after the barrier one warp adds the parts in index order.  1.6 us on
// 148 CTAs, of which the barrier is 1.25.  (Every CTA polling every CTA's part directly, without a
// counter, takes 3 us: the polls of 148 SMs pile up on the same lines.)  `parts`: [2][K][gridDim.x], two
// buffers in turn -- a CTA writes the sum after next only after all have read this one.
template <int K>
struct GridSum {
    double* parts;
    GridSync& gs;
    double* sh;  // shared, [33 * K]
    unsigned int epoch = 0;
    __device__ GridSum(double* p, GridSync& g, double* s) : parts(p), gs(g), sh(s) {}

    // v: each thread's part in, the grid's sum out (in every thread, the same bits in every CTA).  Only
    // the warps that hold one of the first `busy` threads bring anything (the others' parts are zero).
    __device__ __forceinline__ bool sum(double (&v)[K], int busy)
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = gridDim.x;
        const int bw = min((int)(blockDim.x >> 5), (busy + 31) >> 5);
        double* buf = parts + (size_t)(epoch++ & 1) * K * G;
        if (warp < bw) {
#pragma unroll
            for (int q = 0; q < K; q++) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
                if (lane == 0) sh[q * 32 + warp] = v[q];
            }
        }
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int q = 0; q < K; q++) {
                double t = lane < bw ? sh[q * 32 + lane] : 0.0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (lane == 0) buf[(size_t)q * G + blockIdx.x] = t;
            }
            gs.target += G;
            if (lane == 0) gs.arrive_and_wait();
            __syncwarp();
#pragma unroll
            for (int q = 0; q < K; q++) {
                double a[5], t = 0.0;  // 160 CTAs per round of loads: one round on 148 SMs
                for (int c0 = 0; c0 < G; c0 += 160) {
#pragma unroll
                    for (int u = 0; u < 5; u++)
                        a[u] = c0 + 32 * u + lane < G ? __ldcg(buf + (size_t)q * G + c0 + 32 * u + lane) : 0.0;
                    t += ((a[0] + a[1]) + (a[2] + a[3])) + a[4];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (lane == 0) sh[K * 32 + q] = t;
            }
        } else {
            gs.target += G;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < K; q++) v[q] = sh[K * 32 + q];
        return *gs.ok != 0;
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
