// Host side of the matrix-free Kuhn-grid operators (kuhn.cuh, kuhn25.cuh): the z-marching kernel's
// launch configuration and the operator state a solver keeps.
#pragma once

#include <algorithm>

#include "internal.cuh"
#include "kuhn.cuh"
#include "kuhn25.cuh"
#include "zmarch_grid.h"

namespace msfem {

// the z-marching kernel (kuhn25.cuh): TX x TY hexahedron columns per CTA
template <int FORM, bool SC, class T, int TX, int TY, int MINB, class Epi>
struct KzKernel {
    using L = KzLayout<T, TX, TY, Epi::NE, SC>;
    static constexpr auto kernel_iso = k_kuhn_z<FORM, true, SC, T, TX, TY, MINB, Epi>;
    static constexpr auto kernel_aniso = k_kuhn_z<FORM, false, SC, T, TX, TY, MINB, Epi>;
    inline static int blocks_per_sm = 0;
    inline static uint64_t prepared = 0;
    static cudaError_t prepare()
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const uint64_t bit = 1ull << (dev & 63);
        if (prepared & bit) return cudaSuccess;
        e = cudaFuncSetAttribute(kernel_iso, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::smem);
        if (e != cudaSuccess) return e;
        e = cudaFuncSetAttribute(kernel_aniso, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::smem);
        if (e != cudaSuccess) return e;
        int nb = 0, nb2 = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel_iso, L::THREADS, L::smem);
        if (e != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb2, kernel_aniso, L::THREADS, L::smem);
        if (e != cudaSuccess) return e;
        blocks_per_sm = std::max(std::min(nb, nb2), 1);
        prepared |= bit;
        return cudaSuccess;
    }
    // the CTAs of a launch; prepare() first
    static ZmarchGrid grid(const KuhnView<T>& K, int sms)
    {
        return zmarch_grid(K.nx, K.ny, K.nz, L::OX, L::OY, (int64_t)blocks_per_sm * sms);
    }
    // The bulk copies need 16-byte-aligned sources (and read up to 12 bytes past a vector's last
    // element, so every staged vector carries 16 bytes of slack): refused here, never launched.
    static bool aligned(const void* p) { return ((uintptr_t)p & 15) == 0; }
    static cudaError_t launch(const KuhnView<T>& K, const T* x, const Epi& epi, int sms, int* err, cudaStream_t st)
    {
        cudaError_t e = prepare();
        if (e != cudaSuccess) return e;
        const T* ev[Epi::NE > 0 ? Epi::NE : 1] = {};
        epi.sources(ev);
        bool ok = aligned(x) && aligned(K.fix) && aligned(K.mat) && (SC ? (K.scale && aligned(K.scale)) : !K.scale);
        for (int q = 0; q < Epi::NE; q++) ok = ok && ev[q];
        if (!ok) return cudaErrorMisalignedAddress;
        KzArgs<T> A;
        A.K = K;
        A.x = x;
        A.err = err;
        const ZmarchGrid g = grid(K, sms);
        A.tiles_x = g.tiles_x;
        A.tiles_y = g.tiles_y;
        A.seg_len = g.seg_len;
        A.n_seg = g.n_seg;
        return launch_chained(K.iso ? kernel_iso : kernel_aniso, (unsigned)g.ctas(), L::THREADS, L::smem, st, A, epi);
    }
};

// the pre-scaled z-marching kernel (k_kuhn_zp): x = s u with the eliminated columns zero, staged as
// it is; the grid and segment choice as KzKernel's
template <int FORM, class T, int TX, int TY, int MINB, class Epi>
struct KzpKernel {
    using L = KzpLayout<T, TX, TY, Epi::NE>;
    static constexpr auto kernel_iso = k_kuhn_zp<FORM, true, T, TX, TY, MINB, Epi>;
    static constexpr auto kernel_aniso = k_kuhn_zp<FORM, false, T, TX, TY, MINB, Epi>;
    inline static int blocks_per_sm = 0;
    inline static uint64_t prepared = 0;
    static cudaError_t prepare()
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const uint64_t bit = 1ull << (dev & 63);
        if (prepared & bit) return cudaSuccess;
        e = cudaFuncSetAttribute(kernel_iso, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::smem);
        if (e != cudaSuccess) return e;
        e = cudaFuncSetAttribute(kernel_aniso, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::smem);
        if (e != cudaSuccess) return e;
        int nb = 0, nb2 = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel_iso, L::THREADS, L::smem);
        if (e != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb2, kernel_aniso, L::THREADS, L::smem);
        if (e != cudaSuccess) return e;
        blocks_per_sm = std::max(std::min(nb, nb2), 1);
        prepared |= bit;
        return cudaSuccess;
    }
    // the CTAs of a launch; prepare() first
    static ZmarchGrid grid(const KuhnView<T>& K, int sms)
    {
        return zmarch_grid(K.nx, K.ny, K.nz, L::OX, L::OY, (int64_t)blocks_per_sm * sms);
    }
    // 16-byte-aligned sources with 16 bytes of slack, as KzKernel
    static bool aligned(const void* p) { return ((uintptr_t)p & 15) == 0; }
    static cudaError_t launch(const KuhnView<T>& K, const T* x, const Epi& epi, int sms, int* err, cudaStream_t st)
    {
        cudaError_t e = prepare();
        if (e != cudaSuccess) return e;
        const T* ev[Epi::NE > 0 ? Epi::NE : 1] = {};
        epi.sources(ev);
        bool ok = aligned(x) && aligned(K.fix) && aligned(K.mat);
        for (int q = 0; q < Epi::NE; q++) ok = ok && ev[q];
        if (!ok) return cudaErrorMisalignedAddress;
        KzArgs<T> A;
        A.K = K;
        A.x = x;
        A.err = err;
        const ZmarchGrid g = grid(K, sms);
        A.tiles_x = g.tiles_x;
        A.tiles_y = g.tiles_y;
        A.seg_len = g.seg_len;
        A.n_seg = g.n_seg;
        return launch_chained(K.iso ? kernel_iso : kernel_aniso, (unsigned)g.ctas(), L::THREADS, L::smem, st, A, epi);
    }
};

// one matrix-free operator, checked against the assembled matrix of `sys` at values_version
struct KuhnOperator {
    System* sys = nullptr;
    uint64_t version = 0;
    int form = 0;        // 1 the reference's assembly, 2 the textbook orientation
    bool fp64 = false;   // FP64 unscaled (A) or FP32 Jacobi-scaled (S K S)
    bool scaled = false;
    int sms = 0;
    double check_l2 = 0.0, check_max = 0.0;  // relative distance to the assembled product at set-up
    DBuf<int> err;       // raised by a z-marching launch whose staging wait expired
    DBuf<double> lame64;
    DBuf<float> lame32, scale32;
    KuhnView<double> v64{};
    KuhnView<float> v32{};
};

int kuhn_set_grid(System& s, int nx, int ny, int nz);
int kuhn_operator_build(System& s, int form, bool fp64, bool scaled, KuhnOperator& op);
int kuhn_operator_current(const KuhnOperator& op);
int kuhn_spmv64(KuhnOperator& op, const double* x, double* y, cudaStream_t st);
int kuhn_spmv32(KuhnOperator& op, const float* x, float* y, cudaStream_t st);
// y = S K S x through the pre-scaled kernel (k_kuhn_zp): xh (n + 16 elements, scratch) receives
// s x with the eliminated columns zero first; op.sys set
int kuhn_spmv32_pre(KuhnOperator& op, const float* x, float* xh, float* y, cudaStream_t st);
// MSFEM_ERR_CUDA (and the flag cleared) if a z-marching launch on op raised its staging error
int kuhn_check_err(KuhnOperator& op, cudaStream_t st);

// y = op x through the z-marching kernel
template <class T>
struct EpiStoreZ {
    static constexpr int NE = 0;
    T* y;
    __device__ __forceinline__ bool skip() const { return false; }
    __host__ __device__ __forceinline__ void sources(const T** ev) const { (void)ev; }
    __device__ __forceinline__ void operator()(int64_t g, const T* v, const T* xin, const T (*e)[3])
    {
        (void)xin;
        (void)e;
        y[3 * g] = v[0];
        y[3 * g + 1] = v[1];
        y[3 * g + 2] = v[2];
    }
    __device__ __forceinline__ void finish() {}
};
// The z-marching configurations: 16 x 8 hexahedron columns (15 x 7 owned nodes); FP32 four CTAs per SM,
// FP64 two.  A step is a long chain (six tetrahedra a thread, one barrier), so a grid that does not fill the
// SMs evenly waits for the fullest one; CTAs of four warps divide it finer than those of eight, and on large
// grids four independent CTAs hide each other's barriers better than two, which outweighs the wider overlap of
// the smaller tile.  A smoother step at 24^3, 32^3, 40^3, 64^3, 128^3, us: 16 x 8: 4.7, 5.9, 7.7, 17.5, 93;
// 16 x 16: 5.4, 8.5, 9.3, 19.3, 95; 8 x 8: 5.3, 6.5, 8.4, 20.4, 120; 16 x 6: 4.7, 5.8, 7.7, 17.0, 98; 32 x 8: 4.7, 8.0,
// 8.2, 21.0, 93; 24 x 8: 5.6, 6.5, 8.5, 18.0, 97.
constexpr int kKzTX = 16, kKzTY = 8, kKzMinB = 4, kKzMinB64 = 2;

}  // namespace msfem
