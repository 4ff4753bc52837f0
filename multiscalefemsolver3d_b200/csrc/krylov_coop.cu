// Conjugate gradients, a whole solve in one cooperative launch.
//
// One CTA per SM owns a contiguous range of matrix slices.  The inner products are grid sums
// (GridSum, a barrier too) and every CTA derives the step's scalars itself from the same sums, so nothing
// waits for the host between iterations and there is nothing to capture.  The vector that the product gathers is
// written to global memory by its owners; a CTA then copies the range that its columns span (its
// window) into shared memory once per iteration and gathers there.
//
// Three forms, by what fits the shared memory beside the window:
//  - kResident: the CTA's share of the matrix too, copied once; several warps share a slice, each with
//    every W-th column chunk of its rows.  FP64 PCG forms p = z + beta p while it copies the window,
//    which saves one of its three grid-wide waits;
//  - kPlain: matrix and gathers from global memory, one warp per slice;
//  - kTurns: as kPlain, but the grid takes the rows in turn (large scalar systems, see coop_shape).
// The other vectors are in shared memory as far as they fit, the rest in their global arrays.
//
// What bounds it: small systems the grid-wide waits (about 2 microseconds each), large ones the matrix from L2 or
// HBM.  The launch-per-kernel loops this replaces (two kernels per FP32 iteration, three per FP64 one, replayed as
// CUDA graphs) against this, us per iteration: FP64 PCG, scalar 20^3 16.0 -> 7.2, 60^3 22.3 -> 12.6, 100^3 53.9 ->
// 38, 200^3 469 -> 388; elasticity 20^3 24.8 -> 7.8, 40^3 36.7 -> 20, 128^3 572 -> 520 (CG 505 -> 495); FP32 CG,
// scalar 60^3 14.7 -> 8.6, 100^3 32.2 -> 21.2, 200^3 260 -> 230; elasticity 40^3 24.4 -> 9.1, 128^3 295 -> 277.  What
// was tried and not kept for the streaming form: bulk copies of the slices into per-warp shared-memory rings (15.7
// against 12.1 us, FP32 80^3), columns prefetched one slice ahead (19.3 against 17.4 with everything streamed).
#include <algorithm>
#include <cstring>

#include "internal.cuh"
#include "spmv.cuh"

namespace msfem {
namespace {

enum CoopMode { kResident = 0, kPlain = 1, kTurns = 2 };

constexpr int kResidentThreads = 512;
constexpr int kPlainThreads = 1024;

struct CoopArgs {
    int n, maxiter, stall_limit;
    double tol;        // relative to the first (r, r) (the FP32 inner solve)
    const int2* span;  // columns of each slice (nodes)
    int rows;          // capacity of a CTA
    int window;        // elements of the window buffer (a multiple of 4)
    int W;             // kResident: warps per slice
    int keep;          // kPlain: the part of the matrix left in the L2, of 1024
    int entries;       // kResident: capacity of the matrix share (entries / blocks)
    int in_shared;     // how many of the kernel's listed vectors are in shared memory
    GridBar* bar;
    double* parts;
    KState* S;
};

// one CTA's share of the matrix and its layout in shared memory
template <class VT>
struct Share {
    int s0, s1, row0, nr;  // slices [s0, s1), first row, rows
    int lo, hi;            // window [lo, hi) of unknowns, lo a multiple of 4
    int warp, lane, nw;
    int64_t base;          // first stored entry
    VT* win;               // window, at unknown lo
    VT* q;                 // kResident: the product, W parts per row
    unsigned char* mat;    // kResident: values, then columns
    unsigned char* rest;   // listed vectors
};

template <int MODE, int BS, class VT>
__device__ __forceinline__ Share<VT> share_of(const SellView<VT>& A, const CoopArgs& P, unsigned char* sm, int* s_span)
{
    Share<VT> R;
    R.warp = threadIdx.x >> 5;
    R.lane = threadIdx.x & 31;
    R.nw = blockDim.x >> 5;
    R.rest = sm;
    if constexpr (MODE == kTurns) {
        R.row0 = 0;
        R.nr = P.n;
        return R;
    }
    R.s0 = (int)((int64_t)A.n_slices * blockIdx.x / gridDim.x);
    R.s1 = (int)((int64_t)A.n_slices * (blockIdx.x + 1) / gridDim.x);
    R.row0 = R.s0 * kSlice * BS;
    R.nr = min((R.s1 - R.s0) * kSlice * BS, max(0, P.n - R.row0));
    R.base = A.sp[R.s0];
    if constexpr (MODE != kResident) return R;
    if (threadIdx.x < 2) s_span[threadIdx.x] = threadIdx.x == 0 ? 0x7fffffff : -1;
    __syncthreads();
    for (int k = R.s0 + threadIdx.x; k < R.s1; k += blockDim.x) {
        const int2 c = P.span[k];
        atomicMin(&s_span[0], c.x);
        atomicMax(&s_span[1], c.y);
    }
    __syncthreads();
    R.lo = s_span[1] < 0 ? 0 : s_span[0] * BS & ~3;
    R.hi = (s_span[1] + 1) * BS;
    R.win = reinterpret_cast<VT*>(sm);
    R.q = R.win + P.window;
    R.mat = reinterpret_cast<unsigned char*>(R.q + (size_t)P.W * P.rows);
    constexpr int per = BS == 1 ? 1 : 9;
    const int count = (int)(A.sp[R.s1] - R.base);
    unsigned char* cols = R.mat + sizeof(VT) * per * (size_t)P.entries;
    // whole slices: every array starts and ends on 16 bytes
    auto copy = [&](const void* from, unsigned char* to, size_t bytes) {
        for (int i = threadIdx.x; i < (int)(bytes / 16); i += blockDim.x)
            reinterpret_cast<int4*>(to)[i] = __ldcs(reinterpret_cast<const int4*>(from) + i);
    };
    copy(A.val + R.base * per, R.mat, sizeof(VT) * per * (size_t)count);
    if (BS == 1 && A.col16) copy(A.col16 + R.base, cols, 2 * (size_t)count);
    else copy(A.col + R.base, cols, 4 * (size_t)count);
    R.rest = cols + (BS == 1 && A.col16 ? 2 : 4) * (size_t)P.entries;
    return R;
}

// listed vector q: in shared memory when it is among the first `in_shared`, else its rows of the
// caller's global array
template <class VT>
__device__ __forceinline__ VT* place(const Share<VT>& R, const CoopArgs& P, int q, VT* global)
{
    return q < P.in_shared ? reinterpret_cast<VT*>(R.rest) + (size_t)q * P.rows : global + R.row0;
}

__device__ __forceinline__ void load4(const double* p, double (&v)[4])
{
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(p));
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[2]), "=d"(v[3]) : "l"(p + 2));
}
__device__ __forceinline__ void load4(const float* p, float (&v)[4])
{
    asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "l"(p));
}

// window = a + beta b (b null: a alone) for every unknown the CTA's columns span, in batches of
// independent 16-byte (32-byte) loads; a and b are vectors that other CTAs wrote before the last barrier
template <bool TWO, class VT>
__device__ __forceinline__ void fill_window(const Share<VT>& R, const VT* a, const VT* b, VT beta)
{
    constexpr int U = sizeof(VT) == 4 ? 8 : 2;
    const int step = 4 * (int)blockDim.x;
    for (int i0 = R.lo + 4 * (int)threadIdx.x; i0 < R.hi; i0 += U * step) {
        VT v[U][4];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u * step < R.hi) load4(a + i0 + u * step, v[u]);
        if constexpr (TWO) {
            VT w[U][4];
#pragma unroll
            for (int u = 0; u < U; u++)
                if (i0 + u * step < R.hi) load4(b + i0 + u * step, w[u]);
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int k = 0; k < 4; k++) v[u][k] = fma(beta, w[u][k], v[u][k]);
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u * step < R.hi) {
                VT* to = R.win + (i0 + u * step - R.lo);
                if constexpr (sizeof(VT) == 4) {
                    *reinterpret_cast<float4*>(to) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
                } else {
                    *reinterpret_cast<double2*>(to) = make_double2(v[u][0], v[u][1]);
                    *reinterpret_cast<double2*>(to + 2) = make_double2(v[u][2], v[u][3]);
                }
            }
    }
}

// a thread's first row, and the step to its next: within the CTA's range, kTurns over the grid
template <int MODE>
__device__ __forceinline__ int first_row()
{
    return MODE == kTurns ? blockIdx.x * blockDim.x + threadIdx.x : threadIdx.x;
}
template <int MODE>
__device__ __forceinline__ int row_step()
{
    return MODE == kTurns ? gridDim.x * blockDim.x : blockDim.x;
}

// f(row) for every row of the thread.  The product of 3x3 blocks uses all 64 registers that 1024 threads leave, so
// its kernels read the step anew (kept in a register through the product it costs the overlap of the matrix loads:
// 128^3, us an iteration, CG 543 against 495, FP32 319 against 277); scalar ones keep it (PCG 140^3: 105 against
// 114).
template <int MODE, int BS, class F>
__device__ __forceinline__ void each_row(int nr, int step, F&& f)
{
    if constexpr (BS == 3) {
        for (int i = threadIdx.x; i < nr; i += blockDim.x) f(i);
    } else {
        for (int i = first_row<MODE>(); i < nr; i += step) f(i);
    }
}

// f(row, u) in batches of U rows per thread: `load` reads the vectors of row i into slot u, `use` forms
// and stores the new ones -- the loads of a batch are in flight together whatever the arrays alias
template <int MODE, int U, class L, class F>
__device__ __forceinline__ void for_rows(int nr, L&& load, F&& use)
{
    const int step = row_step<MODE>();
    for (int i0 = first_row<MODE>(); i0 < nr; i0 += U * step) {
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u * step < nr) load(i0 + u * step, u);
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u * step < nr) use(i0 + u * step, u);
    }
}

// four values of one lane's chunk from shared memory
__device__ __forceinline__ void chunk_values(const float* p, float (&v)[4])
{
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x;
    v[1] = q.y;
    v[2] = q.z;
    v[3] = q.w;
}
__device__ __forceinline__ void chunk_values(const double* p, double (&v)[4])
{
    const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
}

// chunks sub, sub + step, ... of a scalar slice of `chunks` whose entries lie in shared memory times the
// window; row: the lane's row (clamped), wrow: the window at that row
template <class VT>
__device__ __forceinline__ VT slice_row(const VT* val, const int16_t* c16, const int32_t* c32, int chunks, int sub,
                                        int step, int lane, const VT* wrow, const VT* w0)
{
    VT acc = 0;
#pragma unroll 4
    for (int k = sub; k < chunks; k += step) {
        const int e = (k * kSlice + lane) * kChunk;
        VT v[4];
        chunk_values(val + e, v);
        if (c16) {
            const int2 d = *reinterpret_cast<const int2*>(c16 + e);
            acc += v[0] * wrow[(int)(short)(d.x & 0xffff)];
            acc += v[1] * wrow[(int)(short)((unsigned)d.x >> 16)];
            acc += v[2] * wrow[(int)(short)(d.y & 0xffff)];
            acc += v[3] * wrow[(int)(short)((unsigned)d.y >> 16)];
        } else {
            const int4 d = *reinterpret_cast<const int4*>(c32 + e);
            acc += v[0] * w0[d.x];
            acc += v[1] * w0[d.y];
            acc += v[2] * w0[d.z];
            acc += v[3] * w0[d.w];
        }
    }
    return acc;
}

// kResident: q[(ls * W + sub) * 32 BS + row in slice] = the part of that row's product
template <int BS, class VT>
__device__ __forceinline__ void resident_product(const SellView<VT>& A, const Share<VT>& R, const CoopArgs& P)
{
    constexpr int per = BS == 1 ? 1 : 9, L = kSlice * BS;
    const VT* val = reinterpret_cast<const VT*>(R.mat);
    const void* cols = R.mat + sizeof(VT) * per * (size_t)P.entries;
    const VT* w0 = R.win - R.lo;
    for (int t = R.warp; t < (R.s1 - R.s0) * P.W; t += R.nw) {
        const int ls = t / P.W, sub = t - ls * P.W, sl = R.s0 + ls;
        const int off = (int)(A.sp[sl] - R.base), w = (int)((A.sp[sl + 1] - A.sp[sl]) >> 5);
        VT* out = R.q + (size_t)t * L;
        if constexpr (BS == 1) {
            const int row = min(sl * kSlice + R.lane, A.n_rows - 1);
            out[R.lane] = slice_row<VT>(val + off, A.col16 ? (const int16_t*)cols + off : nullptr,
                                        (const int32_t*)cols + off, w / kChunk, sub, P.W, R.lane, w0 + row, w0);
        } else {
            VT acc[3] = {0, 0, 0};
#pragma unroll 2
            for (int k = sub; k < w; k += P.W) {
                const int b = off + k * kSlice;
                const VT* x = w0 + 3 * ((const int32_t*)cols)[b + R.lane];
                const VT* v = val + 9 * (size_t)b + R.lane;
                const VT x0 = x[0], x1 = x[1], x2 = x[2];
                acc[0] += v[0] * x0 + v[kSlice] * x1 + v[2 * kSlice] * x2;
                acc[1] += v[3 * kSlice] * x0 + v[4 * kSlice] * x1 + v[5 * kSlice] * x2;
                acc[2] += v[6 * kSlice] * x0 + v[7 * kSlice] * x1 + v[8 * kSlice] * x2;
            }
#pragma unroll
            for (int a = 0; a < 3; a++) out[3 * R.lane + a] = acc[a];
        }
    }
}

// f(row, value) for every row of A v that the CTA owns: kPlain local rows, kTurns (scalar) the system's
template <int MODE, int BS, class VT, class F>
__device__ __forceinline__ void plain_product(const SellView<VT>& A, const Share<VT>& R, int keep, const VT* v, F&& f)
{
    if constexpr (MODE == kTurns) {
        static_assert(BS == 1, "rows in turn: scalar systems");
        for (int sl = blockIdx.x * R.nw + R.warp; sl < A.n_slices; sl += gridDim.x * R.nw) {
            const VT t = sell_row_kept<VT>(A, sl, R.lane, v, false);
            if (const int row = sl * kSlice + R.lane; row < R.nr) f(row, t);
        }
        return;
    }
    const int kept = R.s0 + ((R.s1 - R.s0) * keep + 512) / 1024;
    for (int sl = R.s0 + R.warp; sl < R.s1; sl += R.nw) {
        const int lr = (sl - R.s0) * kSlice * BS + R.lane * BS;
        if constexpr (BS == 1) {
            const VT t = sell_row_kept<VT>(A, sl, R.lane, v, sl < kept);
            if (lr < R.nr) f(lr, t);
        } else {
            VT t[3];
            sell_block_kept<VT>(A, sl, R.lane, v, t, sl < kept);
            if (lr < R.nr)
#pragma unroll
                for (int c = 0; c < 3; c++) f(lr + c, t[c]);
        }
    }
}

// the product of row i: the sum of its parts (kResident) or the value itself
template <int MODE, int BS, class VT>
__device__ __forceinline__ VT row_value(const VT* q, int W, int i)
{
    if constexpr (MODE != kResident) {
        return q[i];
    } else {
        constexpr int L = kSlice * BS;
        const VT* p = q + (size_t)(i / L) * W * L + i % L;
        VT t = p[0];
        for (int k = 1; k < W; k++) t += p[(size_t)k * L];
        return t;
    }
}

constexpr int coop_threads(int mode) { return mode == kResident ? kResidentThreads : kPlainThreads; }

// FP64 (Jacobi-)PCG as in CSSD_Matrix::MSG_PreconditioningSSOR (CSSD_Matrix.h:1336-1362), with
// M = diag(A) or M = I: q = A p, alpha = rz / (p, q); x += alpha p, r -= alpha q; beta from (r, z) with
// z = M^-1 r; p = z + beta p.  gx: the solution; gr: the initial residual; S->tol2: the bound on (r, r).
// kPlain gathers gp; kResident gathers gz and gp / gq in turn (the p of the step before).
template <int MODE, int BS, bool JAC>
__global__ void __launch_bounds__(coop_threads(MODE), 1) k_pcg_coop(SellView<double> A, double* gx, double* gr, double* gp,
                                                                    double* gq, double* gz, const double* dinv, CoopArgs P)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ double sh[2 * 33];
    __shared__ int s_ok, s_span[2];
    constexpr bool RES = MODE == kResident;
    const Share<double> R = share_of<MODE, BS>(A, P, sm, s_span);
    const int T = row_step<MODE>(), tid = threadIdx.x;
    double* r = place(R, P, 0, gr);
    double* p = place(R, P, 1, gp);
    double* x = place(R, P, 2, gx);
    double* d = place(R, P, 3, const_cast<double*>(dinv));
    double* q = MODE != kResident ? place(R, P, 4, gq) : R.q;
    auto scaled = [&](int i, double v) { return JAC ? v * d[i] : v; };
    auto each = [&](auto&& f) { each_row<MODE, BS>(R.nr, T, f); };
    GridSync gs(P.bar, &s_ok);
    GridSum<2> sums(P.parts, gs, sh);
    const double tol2 = P.S->tol2;
    double* pp[2] = {gp, gq};
    double v[2] = {0.0, 0.0};
    if (JAC && P.in_shared > 3)
        each([&](int i) { d[i] = dinv[R.row0 + i]; });
    each([&](int i) {
        const double rv = gr[R.row0 + i], zv = scaled(i, rv);
        r[i] = rv;
        x[i] = gx[R.row0 + i];
        p[i] = RES ? 0.0 : zv;
        gp[R.row0 + i] = RES ? 0.0 : zv;
        if (RES) gz[R.row0 + i] = zv;
        v[0] += rv * zv;
        v[1] += rv * rv;
    });
    bool live = sums.sum(v, R.nr);
    double rz = v[0], rr = v[1], beta = 0.0;
    int iter = 0, done = rr <= tol2 ? 1 : 0, breakdown = 0;
    while (live && !done) {
        double pq[2] = {0.0, 0.0};
        int busy = R.nr;
        if constexpr (RES) {
            const double *z = gz, *po = pp[iter & 1];
            double* pn = pp[(iter + 1) & 1];
            fill_window<true>(R, z, po, beta);
            each([&](int i) {
                const double pv = fma(beta, p[i], scaled(i, r[i]));
                p[i] = pv;
                pn[R.row0 + i] = pv;
            });
            __syncthreads();
            resident_product<BS>(A, R, P);
            __syncthreads();
            each([&](int i) { pq[0] += p[i] * row_value<MODE, BS>(q, P.W, i); });
        } else {
            if (!(live = gs.sync())) break;  // the gathered p
            busy = T;
            auto take = [&](int i, double t) {
                q[i] = t;
                pq[0] += p[i] * t;
            };
            plain_product<MODE, BS>(A, R, P.keep, (const double*)gp, take);
        }
        if (!(live = sums.sum(pq, busy))) break;
        if (pq[0] == 0.0 || pq[0] != pq[0]) {
            breakdown = 1;
            done = 1;
            break;
        }
        const double alpha = rz / pq[0];
        v[0] = v[1] = 0.0;
        each([&](int i) {
            x[i] += alpha * p[i];
            const double rv = r[i] - alpha * row_value<MODE, BS>(q, P.W, i);
            r[i] = rv;
            const double zv = scaled(i, rv);
            if (RES) gz[R.row0 + i] = zv;
            v[0] += rv * zv;
            v[1] += rv * rv;
        });
        if (!(live = sums.sum(v, R.nr))) break;
        beta = v[0] / rz;
        rz = v[0];
        rr = v[1];
        iter++;
        if (rr <= tol2) done = 1;
        else if (iter >= P.maxiter) done = 2;
        else if (rr != rr) {
            breakdown = 1;
            done = 3;
        }
        if (!RES && !done)
            each([&](int i) {
                const double pv = fma(beta, p[i], scaled(i, r[i]));
                if (MODE != kTurns) p[i] = pv;
                gp[R.row0 + i] = pv;
            });
    }
    if (P.in_shared > 2)
        each([&](int i) { gx[R.row0 + i] = x[i]; });
    if (live && blockIdx.x == 0 && tid == 0) {
        P.S->rz = rz;
        P.S->rr = rr;
        P.S->iter = iter;
        P.S->breakdown = breakdown;
        P.S->done = done;
    }
}

// FP32 CG on the Jacobi-scaled matrix from x = 0 in the Chronopoulos-Gear arrangement, one reduction
// per iteration:
//   w = A r,  gamma = (r, r),  delta = (w, r)
//   beta = gamma / gamma_old,  alpha = gamma / (delta - beta gamma / alpha_old)
//   p = r + beta p,  s = w + beta s,  x += alpha p,  r -= alpha s
// gr: the right-hand side on entry and the gathered residual; gx: the solution.
template <int MODE, int BS>
__global__ void __launch_bounds__(coop_threads(MODE), 1) k_cg2_coop(SellView<float> A, float* gx, float* gr, float* gw,
                                                                    float* gp, float* gsv, CoopArgs P)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ double sh[2 * 33];
    __shared__ int s_ok, s_span[2];
    const Share<float> R = share_of<MODE, BS>(A, P, sm, s_span);
    const int T = row_step<MODE>(), tid = threadIdx.x;
    float* r = place(R, P, 0, gr);
    float* s = place(R, P, 1, gsv);
    float* p = place(R, P, 2, gp);
    float* x = place(R, P, 3, gx);
    float* w = MODE != kResident ? place(R, P, 4, gw) : R.q;
    auto each = [&](auto&& f) { each_row<MODE, BS>(R.nr, T, f); };
    GridSync gs(P.bar, &s_ok);
    GridSum<2> sums(P.parts, gs, sh);
    each([&](int i) {
        r[i] = gr[R.row0 + i];
        x[i] = 0.0f;
        p[i] = 0.0f;
        s[i] = 0.0f;
    });
    __syncthreads();
    double gamma = 0.0, alpha_old = 1.0, gamma_old = 0.0, rr_min = 0.0, tol2 = 0.0;
    int iter = 0, stall = 0, done = 0;
    bool live = true;
    for (bool first = true;; first = false) {
        double v[2] = {0.0, 0.0};
        int busy = R.nr;
        if constexpr (MODE == kResident) {
            fill_window<false>(R, (const float*)gr, (const float*)nullptr, 0.0f);
            __syncthreads();
        }
        auto take = [&](int i, float t) {
            const double rv = (double)r[i];
            w[i] = t;
            v[0] += rv * rv;
            v[1] += (double)t * rv;
        };
        if constexpr (MODE == kResident) {
            resident_product<BS>(A, R, P);
            __syncthreads();
            each([&](int i) {
                const double rv = (double)r[i];
                v[0] += rv * rv;
                v[1] += (double)row_value<MODE, BS>(w, P.W, i) * rv;
            });
        } else {
            busy = T;
            plain_product<MODE, BS>(A, R, P.keep, (const float*)gr, take);
        }
        if (!(live = sums.sum(v, busy))) break;
        gamma = v[0];
        if (first) {
            tol2 = P.tol * P.tol * gamma;
            rr_min = gamma;
        } else if (gamma < 0.98 * rr_min) {
            rr_min = gamma;
            stall = 0;
        } else {
            stall++;
        }
        const double beta = first ? 0.0 : gamma / gamma_old;
        const double den = first ? v[1] : v[1] - beta * gamma / alpha_old;
        const double alpha = gamma / den;
        if (gamma <= tol2) done = 1;
        else if (iter >= P.maxiter) done = 2;
        else if (!(den != 0.0) || den != den || gamma != gamma) done = 3;  // breakdown
        else if (stall >= P.stall_limit) done = 4;  // FP32 attainable accuracy reached
        if (done) break;
        iter++;
        gamma_old = gamma;
        alpha_old = alpha;
        const float al = (float)alpha, be = (float)beta;
        {
            float rs[4], ps[4], ws[4], ss[4], xs[4];
            for_rows<MODE, MODE == kResident || BS == 3 ? 1 : 4>(
                R.nr,
                [&](int i, int u) {
                    rs[u] = r[i];
                    ps[u] = p[i];
                    ws[u] = row_value<MODE, BS>(w, P.W, i);
                    ss[u] = s[i];
                    xs[u] = x[i];
                },
                [&](int i, int u) {
                    const float pi = rs[u] + be * ps[u];
                    const float si = ws[u] + be * ss[u];
                    p[i] = pi;
                    s[i] = si;
                    x[i] = xs[u] + al * pi;
                    const float rv = rs[u] - al * si;
                    if (MODE != kTurns) r[i] = rv;
                    gr[R.row0 + i] = rv;
                });
        }
        if (!(live = gs.sync())) break;  // the gathered r
    }
    if (P.in_shared > 3)
        each([&](int i) { gx[R.row0 + i] = x[i]; });
    if (live && blockIdx.x == 0 && tid == 0) {
        P.S->rr = gamma;
        P.S->iter = iter;
        P.S->breakdown = done == 3;
        P.S->done = done;
    }
}

// The launch shape: one CTA per SM (fewer where there are fewer slices), the form and the vectors in
// shared memory by what fits (see the top).
struct CoopShape {
    int mode, G, threads;
    size_t smem;
};

int coop_shape(System& s, int vectors, size_t width, bool col16, CoopArgs& P, CoopShape* c)
{
    int dev = 0, sms = 0, most = 0;
    MSFEM_CK(cudaGetDevice(&dev));
    MSFEM_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MSFEM_CK(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const int n_slices = s.sell.n_slices, bs = s.bs;
    c->G = std::max(1, std::min(sms, n_slices));
    const int per = (n_slices + c->G - 1) / c->G;
    P.rows = per * kSlice * bs;
    P.span = s.sell.span.p;
    P.window = (int)std::min<int64_t>(((int64_t)s.sell.max_span * bs + 11) / 4 * 4, 1 << 20);
    const size_t room = (size_t)most - 4096, one = width * (size_t)P.rows;
    const size_t window = width * (size_t)P.window, cw = bs == 1 && col16 ? 2 : 4;
    // resident: the widest slice bounds every share
    const size_t entries = (size_t)per * s.sell.max_width * kSlice;
    const int units = bs == 1 ? s.sell.max_width / kChunk : s.sell.max_width;
    P.W = std::max(1, std::min(units, kResidentThreads / 32 / per));
    const size_t need = window + one * P.W + entries * (bs == 1 ? width : 9 * width) + entries * cw;
    if (need + one * (vectors - 1) <= room) {
        c->mode = kResident;
        c->threads = std::min(kResidentThreads, std::max(per * P.W * 32, 128));
        P.entries = (int)entries;
        P.in_shared = vectors - 1;  // all but the product, which has its own place
        c->smem = need + one * P.in_shared;
        return MSFEM_OK;
    }
    int l2 = 0;
    MSFEM_CK(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev));
    // the window of a CTA's range, of which a few columns may lie far away; without a spatial order there is none
    const double window_of_range = s.sell.slice_span + (double)per * kSlice;
    const bool scattered = s.sell.scattered;
    P.W = 1;
    // The CTAs sweep their ranges at the same time, each behind its own window of the gathered vector.  Where the
    // windows together exceed the L2, the grid takes the rows in turn, so that one window serves all.  Scalar FP64,
    // us an iteration, ranges / turns: CG 160^3 175 / 176, 200^3 387 / 375, 240^3 683 / 635; 3x3 blocks, whose matrix
    // is nine times the window's traffic, are faster by ranges (CG 128^3 495 / 515), and so are scattered columns,
    // whose windows are the whole vector either way (CG 200^3 660 / 695).
    if (bs == 1 && !scattered && c->G * window_of_range * width > l2) {
        c->mode = kTurns;
        c->threads = kPlainThreads;
        P.in_shared = 0;
        c->smem = 0;
        return MSFEM_OK;
    }
    c->mode = kPlain;
    P.keep = keep_share(s, width);
    c->threads = std::min(kPlainThreads, std::max(per * 32, 256));
    // shared memory beyond this leaves the gathers too little L1 (FP64 at 100^3: 45 us an iteration with four
    // vectors, 223 KB, in shared memory, 38 with three; FP32 at 140^3: 69 with three, 63 with two), and scattered
    // columns need more of it (elasticity 64^3 in random order, CG: four 92 us, three 77, two and one 67; 80^3: two
    // 171, one 130, none 125; FP32 128^3: one 415, none 345)
    P.in_shared = (int)std::min<size_t>(vectors, std::min<size_t>(room, (scattered ? 64 : 176) << 10) / one);
    c->smem = one * P.in_shared;
    return MSFEM_OK;
}

int coop_launch(System& s, const void* kernel, const CoopShape& c, CoopArgs& P, void** args)
{
    size_t room = 0;
    MSFEM_TRY(open_shared_memory(kernel, &room));
    const size_t bytes = 16 + sizeof(double) * 4 * (size_t)c.G;
    MSFEM_TRY(s.coop.alloc(bytes));
    MSFEM_CK(cudaMemsetAsync(s.coop.p, 0, 16, s.stream));
    P.bar = reinterpret_cast<GridBar*>(s.coop.p);
    P.parts = reinterpret_cast<double*>(s.coop.p + 16);
    P.n = s.n_rows;
    P.S = s.kstate.p;
    MSFEM_CK(cudaLaunchCooperativeKernel(kernel, dim3(c.G), dim3(c.threads), args, c.smem, s.stream));
    s.launches += 1;
    GridBar h{};
    MSFEM_CK(cudaMemcpyAsync(&h, s.coop.p, sizeof(h), cudaMemcpyDeviceToHost, s.stream));
    MSFEM_TRY(read_state(s));
    if (h.abort) {
        set_error("CG: a grid-wide wait expired");
        return MSFEM_ERR_CUDA;
    }
    return MSFEM_OK;
}

template <bool JAC>
const void* pcg_kernel(int mode, int bs)
{
    if (mode == kTurns) return (const void*)k_pcg_coop<kTurns, 1, JAC>;
    if (mode == kResident && bs == 1) return (const void*)k_pcg_coop<kResident, 1, JAC>;
    if (mode == kResident) return (const void*)k_pcg_coop<kResident, 3, JAC>;
    return bs == 1 ? (const void*)k_pcg_coop<kPlain, 1, JAC> : (const void*)k_pcg_coop<kPlain, 3, JAC>;
}

const void* cg2_kernel(int mode, int bs)
{
    if (mode == kTurns) return (const void*)k_cg2_coop<kTurns, 1>;
    if (mode == kResident && bs == 1) return (const void*)k_cg2_coop<kResident, 1>;
    if (mode == kResident) return (const void*)k_cg2_coop<kResident, 3>;
    return bs == 1 ? (const void*)k_cg2_coop<kPlain, 1> : (const void*)k_cg2_coop<kPlain, 3>;
}

}  // namespace

int open_shared_memory(const void* kernel, size_t* room)
{
    int dev = 0, most = 0;
    cudaFuncAttributes a{};
    MSFEM_CK(cudaGetDevice(&dev));
    MSFEM_CK(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    MSFEM_CK(cudaFuncGetAttributes(&a, kernel));
    *room = (size_t)most - a.sharedSizeBytes;
    MSFEM_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*room));
    return MSFEM_OK;
}

int pcg64_coop(System& s, bool jacobi, double* x, double* r, double* p, double* q, double* z, int maxiter)
{
    SellView<double> A = sell_view<double>(s);
    CoopArgs P{};
    P.maxiter = maxiter;
    CoopShape c;
    MSFEM_TRY(coop_shape(s, 5, sizeof(double), A.col16 != nullptr, P, &c));
    const double* dinv = s.dinv64.p;
    void* args[] = {&A, &x, &r, &p, &q, &z, &dinv, &P};
    return coop_launch(s, jacobi ? pcg_kernel<true>(c.mode, s.bs) : pcg_kernel<false>(c.mode, s.bs), c, P, args);
}

int cg32_coop(System& s, float* x, float* r, float* w, float* p, float* sv, double tol, int maxiter, int stall_limit)
{
    // 16-bit column deltas where they fit: 21.2 us an iteration at 100^3 against 30.1 with 32-bit columns
    const int tuned = s.sell.fp32_col16;
    s.sell.fp32_col16 = s.sell.col16.p ? 1 : 0;
    SellView<float> A = sell_view<float>(s);
    s.sell.fp32_col16 = tuned;
    CoopArgs P{};
    P.maxiter = maxiter;
    P.tol = tol;
    P.stall_limit = stall_limit;
    CoopShape c;
    MSFEM_TRY(coop_shape(s, 5, sizeof(float), A.col16 != nullptr, P, &c));
    void* args[] = {&A, &x, &r, &w, &p, &sv, &P};
    return coop_launch(s, cg2_kernel(c.mode, s.bs), c, P, args);
}

}  // namespace msfem
