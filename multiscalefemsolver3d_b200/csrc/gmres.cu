// Restarted GMRES(m) on the GPU, right-preconditioned by diag(A).
//
// The reference's compiled GMRES (CSSD_Matrix.h:1774-1989) has no caller and a
// fixed depth of 5; its legacy GMRS (Library/GMRES/7_gmres.for:95-222) is a
// restarted GMRES(M) with Givens rotations and a back substitution.  This is
// that method laid out for the GPU:
//   * Arnoldi with classical Gram-Schmidt applied twice (CGS2): the j+1
//     projections of a step are computed together and removed together,
//     instead of 2(j+1) dependent passes;
//   * the Hessenberg column, its Givens rotations and the residual estimate
//     |g_{j+1}| are updated on the device: the host waits once per solve;
//   * x += M^-1 V y is one fused pass after the cycle.
// Stopping test: |g_{j+1}| <= tol * ||F|| (the true residual norm in exact
// arithmetic for right preconditioning).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "devutil.cuh"
#include "internal.cuh"
#include "spmv.cuh"

namespace msfem {
namespace {

// One cooperative launch runs the whole solve -- every Arnoldi step, restart and residual.  CTA c owns
// a contiguous range of matrix slices and keeps its rows of the work vector (and, where they fit, of
// every basis vector) in shared memory, so an Arnoldi step reads the matrix and the gathered vector;
// its three reductions (the two Gram-Schmidt projections and the norm) are grid barriers.  Every CTA
// keeps the rotations and the residual estimate itself, from the same sums in the same order; CTA 0
// keeps the Hessenberg matrix.  The launch-per-kernel cycle this replaces was bound by its launches
// and by the last block's serial reduction of j + 1 sums: with restart 50 an Arnoldi step took 134 us
// at 72,522 unknowns, 160 us at 282,962 and 306 us at 949,567 (FP32 basis); here 17, 42 and 142 us.
// With the basis in global memory 1024 threads beat 512 (47 against 55 us at 282,962 unknowns, FP64 56
// against 89): more loads in flight per SM; in shared memory 512 leave room for the basis.

struct GmCoop {
    int n, m, maxiter, rows;  // rows: capacity of a CTA (slices * 32 * bs)
    int keep;                 // part of the matrix left in the L2, of 1024
    double tol;
    const double* dinv;       // right preconditioner diag(A)^-1, or null
    void* x;                  // solution, VT
    const void* b;            // right-hand side, VT
    int zero_start;           // x = 0 on entry
    void* gather[2];          // [n] each, VT
    double* partial;          // [2 m + 4][gridDim.x]
    void* V;                  // [m + 1][n] basis, VT, when the CTAs' shares do not fit shared memory
    void* w;                  // [n] work vector, VT, when it does not fit either
    double* H;                // [m (m + 1) / 2] packed upper triangle, column j at j (j + 1) / 2
    double* y;                // [m]
    double* out;              // [0] iterations, [1] cycles, [2] |g|^2 at the end, [3] done, [4] ||b||^2
    GridBar* bar;
};

// sums of `count` values over the grid: the CTA's value q (written by the caller into vals[q parts ..], shared,
// as `parts` numbers) -> sums[q] (shared), the CTAs added in index order by lanes and a butterfly
__device__ __forceinline__ bool grid_sums(GridSync& gs, double* partial, const double* vals, double* sums, int count,
                                          int parts = 1)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, G = gridDim.x;
    __syncthreads();
    for (int q = threadIdx.x; q < count; q += blockDim.x) {
        double t = vals[q * parts];
        for (int p = 1; p < parts; p++) t += vals[q * parts + p];
        partial[(size_t)q * G + blockIdx.x] = t;
    }
    if (!gs.sync()) return false;
    for (int q = warp; q < count; q += nw) {
        const double* p = partial + (size_t)q * G;
        double a[5], t = 0.0;  // 160 CTAs per round of loads: one round on 148 SMs
        for (int c0 = 0; c0 < G; c0 += 160) {
#pragma unroll
            for (int u = 0; u < 5; u++) a[u] = c0 + 32 * u + lane < G ? __ldcg(p + c0 + 32 * u + lane) : 0.0;
            t += ((a[0] + a[1]) + (a[2] + a[3])) + a[4];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) sums[q] = t;
    }
    __syncthreads();
    return true;
}

// where a CTA's rows of the basis and of the work vector are: both in shared memory, the work vector there, neither
enum GmForm { kBasisShared, kWorkShared, kAllGlobal };

// Restarts of up to kFew vectors with the basis in global memory have passes of their own (FEW): with a vector to a
// warp most warps idle, and with a row to a thread too little is in flight.  us a step at restart 5, 10, 16, without
// / with them (the launch-per-kernel cycle): elasticity 128^3 FP64 966, 980, 986 / 686, 710, 780 (797, 895, 1063),
// FP32 706, 724, 728 / 422, 468, 546 (486, 594, 752); scalar 140^3 FP64 260, 283, 295 / 159, 181, 217 (230, 292,
// 377).  More vectors fill the warps by themselves (restart 20 at 128^3 FP64: 1031, launch per kernel 1166).
constexpr int kFew = 16;

template <class VT, int FORM, bool FEW>
__global__ void __launch_bounds__(FORM == kBasisShared ? 512 : 1024, 1) k_gm_coop(SellView<VT> A, GmCoop P)
{
    constexpr bool VS = FORM == kBasisShared;
    // the work vector holds values rounded to VT: as FP64, which spares the conversions, except where its traffic
    // counts
    using WT = std::conditional_t<FORM == kAllGlobal && FEW, VT, double>;
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ int s_ok;
    __shared__ double s_warp[32], s_one[1], s_norm[1];
    __shared__ double s_state[4];  // [0] |g_{j+1}|, [1] stop code
    const int m = P.m, tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
    // shared memory: FP64 small arrays, then the basis rows and the work rows
    double* h1 = reinterpret_cast<double*>(sm);  // own partial dots, those of a vector in up to a part per warp
    double* h2 = h1 + m + 1 + 32;                // summed: first projection
    double* h3 = h2 + m + 1;                     // summed: second projection
    double* cs = h3 + m + 1;
    double* sn = cs + m;
    double* g = sn + m;
    double* y = g + m + 1;
    WT* w;
    VT* V = (VT*)P.V;
    int64_t ldv = P.n;
    GridSync gs(P.bar, &s_ok);
    const int G = gridDim.x;
    const int s0 = (int)((int64_t)A.n_slices * blockIdx.x / G), s1 = (int)((int64_t)A.n_slices * (blockIdx.x + 1) / G);
    const int row0 = s0 * kSlice * A.bs, kept = s0 + ((s1 - s0) * P.keep + 512) / 1024;
    const int nr = min((s1 - s0) * kSlice * A.bs, max(0, P.n - row0));  // this CTA's rows
    if (VS) {
        V = reinterpret_cast<VT*>(y + m + P.rows);
        ldv = P.rows;
    } else {
        V += row0;
    }
    if constexpr (FORM == kAllGlobal) w = (WT*)P.w + row0;
    else w = y + m;
    VT* x = reinterpret_cast<VT*>(P.x);
    const VT* b = reinterpret_cast<const VT*>(P.b);

    // w = scale * A v on the CTA's rows
    auto product = [&](const VT* v, double scale) {
        for (int sl = s0 + warp; sl < s1; sl += nw) {
            const int lr = (sl - s0) * kSlice * A.bs + lane * A.bs;
            if (A.bs == 1) {
                const VT t = sell_row_kept<VT>(A, sl, lane, v, sl < kept);
                if (lr < nr) w[lr] = (WT)(VT)(t * (VT)scale);
            } else {
                VT t[3];
                sell_block_kept<VT>(A, sl, lane, v, t, sl < kept);
                if (lr < nr)
                    for (int c = 0; c < 3; c++) w[lr + c] = (WT)(VT)(t[c] * (VT)scale);
            }
        }
        __syncthreads();
    };
    // (w, w) over the grid into s_norm[0]
    auto norm2 = [&](double* part) -> bool {
        double t = 0.0;
        for (int r = tid; r < nr; r += T) t += (double)w[r] * (double)w[r];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) s_warp[warp] = t;
        __syncthreads();
        if (tid == 0) {
            double u = 0.0;
            for (int k = 0; k < nw; k++) u += s_warp[k];
            s_one[0] = u;
        }
        return grid_sums(gs, part, s_one, s_norm, 1);
    };
    // the vector the next product gathers: w, through the right preconditioner
    auto publish = [&](VT* to) {
        for (int r = tid; r < nr; r += T)
            to[row0 + r] = (VT)(P.dinv ? (double)w[r] * P.dinv[row0 + r] : (double)w[r]);
    };
    // h1[i] (+)= (V_i, w) on the CTA's rows [r0, r1), one vector per warp at a time
    auto dots = [&](int j, int r0, int r1, bool add) {
        for (int i = warp; i <= j; i += nw) {
            const VT* v = V + i * ldv;
            double t[4] = {0.0, 0.0, 0.0, 0.0};
            for (int r = r0 + lane; r < r1; r += 128)
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (r + 32 * u < r1) t[u] += (double)v[r + 32 * u] * (double)w[r + 32 * u];
            double q = (t[0] + t[1]) + (t[2] + t[3]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
            if (lane == 0) h1[i] = add ? h1[i] + q : q;
        }
    };
    // w -= sum_i h[i] V_i; with `again`, h1 = the projections of the new w, tile by tile of rows, so
    // that the second read of the basis finds the tile in the L1
    auto remove = [&](const double* h, int j, bool again) {
        for (int r0 = 0; r0 < nr; r0 += T) {
            const int r = r0 + tid;
            if (r < nr) {
                double t[4] = {(double)w[r], 0.0, 0.0, 0.0};
                int i = 0;
                for (; i + 3 <= j; i += 4)
#pragma unroll
                    for (int u = 0; u < 4; u++) t[u] -= h[i + u] * (double)V[(i + u) * ldv + r];
                for (; i <= j; i++) t[0] -= h[i] * (double)V[i * ldv + r];
                w[r] = (WT)(VT)((t[0] + t[1]) + (t[2] + t[3]));
            }
            if (again) {
                __syncthreads();
                dots(j, r0, min(r0 + T, nr), r0 > 0);
            }
        }
        if (again && nr == 0)
            for (int i = tid; i <= j; i += T) h1[i] = 0.0;
        __syncthreads();
    };

    // FEW: nw / nv warps share the rows of each of the nv vectors, a thread keeps four rows in flight, and a vector's
    // sums stay in registers over the tiles; h1[i parts + p] = part p of vector i
    auto few_dots = [&](int nv, int parts, int r0, int r1, double (&t)[4]) {
        const int i = warp / parts, p = warp - i * parts;
        if (i >= nv) return;
        const VT* v = V + i * ldv;
        for (int r = r0 + 128 * p + lane; r < r1; r += 128 * parts)
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (r + 32 * u < r1) t[u] += (double)v[r + 32 * u] * (double)w[r + 32 * u];
    };
    auto few_dots_end = [&](double (&t)[4]) {
        double q = (t[0] + t[1]) + (t[2] + t[3]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
        if (lane == 0) h1[warp] = q;
    };
    auto few_remove = [&](const double* h, int nv, int parts, bool again) {
        constexpr int U = 4;
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        for (int r0 = 0; r0 < nr; r0 += U * T) {
            double t[U];
#pragma unroll
            for (int u = 0; u < U; u++) t[u] = r0 + u * T + tid < nr ? (double)w[r0 + u * T + tid] : 0.0;
            for (int i = 0; i < nv; i++)
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (r0 + u * T + tid < nr) t[u] -= h[i] * (double)V[i * ldv + r0 + u * T + tid];
#pragma unroll
            for (int u = 0; u < U; u++)
                if (r0 + u * T + tid < nr) w[r0 + u * T + tid] = (WT)(VT)t[u];
            if (again) {
                __syncthreads();
                few_dots(nv, parts, r0, min(r0 + U * T, nr), s);
            }
        }
        if (again) few_dots_end(s);
        __syncthreads();
    };

    double* part1 = P.partial;
    double* part2 = part1 + (size_t)(m + 1) * G;
    double* part3 = part2 + (size_t)(m + 1) * G;
    double* part4 = part3 + G;
    int iter = 0, cycles = 0, done = 0;
    for (int r = tid; r < nr; r += T) w[r] = b[row0 + r];
    __syncthreads();
    if (!norm2(part4)) return;
    const double bb = s_norm[0], tol2 = P.tol * P.tol * bb;
    double res2 = bb;
    bool zero = P.zero_start != 0;
    for (;;) {
        // r = b - A x, its norm
        __syncthreads();
        if (!zero) {  // else w holds b
            product(x, 1.0);
            for (int r = tid; r < nr; r += T) w[r] = (WT)(VT)((double)b[row0 + r] - (double)w[r]);
        }
        zero = false;
        __syncthreads();
        publish((VT*)P.gather[0]);
        if (!norm2(part3)) return;
        res2 = s_norm[0];
        if (res2 <= tol2 || done || iter >= P.maxiter || !(res2 == res2)) break;
        cycles++;
        double norm = sqrt(res2);
        for (int i = tid; i <= m; i += T) g[i] = i == 0 ? norm : 0.0;
        if (tid == 0) s_state[1] = 0.0;
        int k = 0;
        for (int j = 0; j < m; j++) {
            const double inv = norm > 0.0 ? 1.0 / norm : 0.0;
            for (int r = tid; r < nr; r += T) V[j * ldv + r] = (VT)((double)w[r] * inv);
            __syncthreads();
            product((const VT*)P.gather[j & 1], inv);
            if constexpr (FEW) {
                const int nv = j + 1, parts = nw / nv;
                double t[4] = {0.0, 0.0, 0.0, 0.0};
                few_dots(nv, parts, 0, nr, t);
                few_dots_end(t);
                if (!grid_sums(gs, part1, h1, h2, nv, parts)) return;
                few_remove(h2, nv, parts, true);
                if (!grid_sums(gs, part2, h1, h3, nv, parts)) return;
                few_remove(h3, nv, parts, false);
            } else {
                dots(j, 0, nr, false);
                if (!grid_sums(gs, part1, h1, h2, j + 1)) return;
                remove(h2, j, true);
                if (!grid_sums(gs, part2, h1, h3, j + 1)) return;
                remove(h3, j, false);
            }
            publish((VT*)P.gather[(j + 1) & 1]);
            if (!norm2(part3)) return;
            norm = sqrt(s_norm[0]);
            if (tid == 0) {
                double* Hj = P.H + (size_t)j * (j + 1) / 2;
                const bool keep = blockIdx.x == 0;
                double a = h2[0] + h3[0];
                for (int i = 0; i < j; i++) {
                    const double nx = h2[i + 1] + h3[i + 1];
                    if (keep) Hj[i] = cs[i] * a + sn[i] * nx;
                    a = -sn[i] * a + cs[i] * nx;
                }
                const double d = sqrt(a * a + norm * norm);
                const double c = d > 0 ? a / d : 1.0, s = d > 0 ? norm / d : 0.0;
                cs[j] = c;
                sn[j] = s;
                if (keep) Hj[j] = d;
                g[j + 1] = -s * g[j];
                g[j] = c * g[j];
                const double res = fabs(g[j + 1]);
                double code = 0.0;
                if (res * res <= tol2 || !(res == res)) code = 1.0;
                else if (norm == 0.0 || d == 0.0) code = 2.0;  // the cycle's space holds the solution
                else if (iter + 1 >= P.maxiter) code = 3.0;
                s_state[0] = res * res;
                s_state[1] = code;
            }
            __syncthreads();
            iter++;
            k = j + 1;
            if (s_state[1] != 0.0) break;
        }
        res2 = s_state[0];
        if (s_state[1] == 1.0) done = 1;
        else if (s_state[1] == 3.0) done = 2;
        // y = R^-1 g, column by column (warp 0 of CTA 0), then x += M^-1 V y on the CTA's rows
        if (blockIdx.x == 0 && warp == 0) {
            for (int i = lane; i < k; i += 32) y[i] = g[i];
            __syncwarp();
            for (int i = k - 1; i >= 0; i--) {
                const double* Hi = P.H + (size_t)i * (i + 1) / 2;
                const double yi = Hi[i] != 0.0 ? y[i] / Hi[i] : 0.0;
                __syncwarp();
                for (int l = lane; l < i; l += 32) y[l] -= Hi[l] * yi;
                if (lane == 0) y[i] = yi;
                __syncwarp();
            }
            for (int i = lane; i < k; i += 32) P.y[i] = y[i];
        }
        if (!gs.sync()) return;
        for (int i = tid; i < k; i += T) y[i] = __ldcg(P.y + i);
        __syncthreads();
        for (int r = tid; r < nr; r += T) {
            double t[4] = {0.0, 0.0, 0.0, 0.0};
            int i = 0;
            for (; i + 3 < k; i += 4)
#pragma unroll
                for (int u = 0; u < 4; u++) t[u] += y[i + u] * (double)V[(i + u) * ldv + r];
            for (; i < k; i++) t[0] += y[i] * (double)V[i * ldv + r];
            const double old = P.zero_start && cycles == 1 ? 0.0 : (double)x[row0 + r];
            x[row0 + r] = (VT)(old + (P.dinv ? P.dinv[row0 + r] : 1.0) * ((t[0] + t[1]) + (t[2] + t[3])));
        }
        if (done) break;
        if (!gs.sync()) return;  // x is gathered by the next residual
    }
    if (P.zero_start && cycles == 0)
        for (int r = tid; r < nr; r += T) x[row0 + r] = (VT)0;
    if (blockIdx.x == 0 && tid == 0) {
        P.out[0] = iter;
        P.out[1] = cycles;
        P.out[2] = res2;
        P.out[3] = done;
        P.out[4] = bb;
    }
}

// The launch: one CTA of 512 threads per SM (fewer where there are fewer slices); the basis goes to
// shared memory while a CTA's share of it fits beside the work vector (restart 50: up to about
// 140,000 unknowns with an FP32 basis).
template <class VT>
struct GmShape {
    const void* kernel;
    int G, rows, threads;
    size_t smem;
    bool w_shared, basis_shared;
    static int make(const SellView<VT>& A, int m, bool scattered, GmShape* out)
    {
        int dev = 0, sms = 0;
        MSFEM_CK(cudaGetDevice(&dev));
        MSFEM_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        const void* kernels[3] = {(const void*)k_gm_coop<VT, kBasisShared, false>,
                                  (const void*)k_gm_coop<VT, kWorkShared, false>,
                                  (const void*)k_gm_coop<VT, kAllGlobal, false>};
        if (m <= kFew) {
            kernels[kWorkShared] = (const void*)k_gm_coop<VT, kWorkShared, true>;
            kernels[kAllGlobal] = (const void*)k_gm_coop<VT, kAllGlobal, true>;
        }
        size_t room[3];
        for (int f = 0; f < 3; f++) MSFEM_TRY(open_shared_memory(kernels[f], &room[f]));
        out->G = std::max(1, std::min(sms, A.n_slices));
        out->rows = (A.n_slices + out->G - 1) / out->G * kSlice * A.bs;
        // the small arrays; the 1 KB holds the parts of h1 too
        const size_t small = sizeof(double) * (4 * (size_t)(m + 1) + 3 * (size_t)m) + 1024;
        const size_t w = sizeof(double) * out->rows, v = sizeof(VT) * (size_t)(m + 1) * out->rows;
        // gathers in no spatial order need some L1 (us a step, basis in shared / global memory: scalar 80^3 in random
        // order, FP64 with restart 5, 202 KB, 110 / 59; 100^3 FP32, 223 KB, 188 / 91; 60^3 FP64 restart 10, 147 KB,
        // 29 / 33)
        const size_t basis_room = std::min<size_t>(room[kBasisShared], scattered ? 164 << 10 : room[kBasisShared]);
        const GmForm form = small + w + v <= basis_room      ? kBasisShared
                            : small + w <= room[kWorkShared] ? kWorkShared
                                                             : kAllGlobal;
        out->basis_shared = form == kBasisShared;
        out->w_shared = form != kAllGlobal;
        out->threads = form == kBasisShared ? 512 : 1024;
        out->smem = small + (out->w_shared ? w : 0) + (out->basis_shared ? v : 0);
        out->kernel = kernels[form];
        return MSFEM_OK;
    }
};

// Runs the solve; P: everything but the workspace fields.  V: [m + 1][n], g0 / g1: [n].  out5 (host)
// receives P.out.
template <class VT>
int gm_coop_run(System& s, GmCoop P, VT* V, VT* g0, VT* g1, double* out5)
{
    SellView<VT> A = sell_view<VT>(s);
    GmShape<VT> shape;
    MSFEM_TRY(GmShape<VT>::make(A, P.m, s.sell.scattered, &shape));
    const size_t np = (size_t)(2 * P.m + 4) * shape.G, nh = (size_t)P.m * (P.m + 1) / 2;
    MSFEM_TRY(s.gm.alloc(8 + np + nh + P.m + (shape.w_shared ? 0 : (size_t)P.n)));
    MSFEM_CK(cudaMemsetAsync(s.gm.p, 0, sizeof(double) * 8, s.stream));
    P.rows = shape.rows;
    // a basis in global memory would push a kept matrix out of the L2 in turn
    P.keep = shape.basis_shared ? keep_share(s, sizeof(VT)) : 0;
    P.V = V;
    P.gather[0] = g0;
    P.gather[1] = g1;
    P.out = s.gm.p;
    P.bar = reinterpret_cast<GridBar*>(s.gm.p + 6);
    P.partial = s.gm.p + 8;
    P.H = P.partial + np;
    P.y = P.H + nh;
    P.w = shape.w_shared ? nullptr : P.y + P.m;
    void* args[] = {&A, &P};
    MSFEM_CK(cudaLaunchCooperativeKernel(shape.kernel, dim3(shape.G), dim3(shape.threads), args, shape.smem, s.stream));
    s.launches += 1;
    double h[8];
    MSFEM_CK(cudaMemcpyAsync(h, s.gm.p, sizeof(h), cudaMemcpyDeviceToHost, s.stream));
    MSFEM_CK(cudaStreamSynchronize(s.stream));
    unsigned int bar[2];
    std::memcpy(bar, &h[6], sizeof(bar));
    if (bar[1]) {
        set_error("GMRES: a grid barrier expired");
        return MSFEM_ERR_CUDA;
    }
    for (int k = 0; k < 5; k++) out5[k] = h[k];
    return MSFEM_OK;
}

}  // namespace

int solve_gmres64(System& s, int m, int maxiter, double tol, int* iters, int* restarts)
{
    if (m < 1 || m > 1000) {
        set_error("GMRES restart depth must be in [1, 1000]");
        return MSFEM_ERR_ARGUMENT;
    }
    const int n = s.n_rows;
    MSFEM_TRY(s.work64.alloc((size_t)(m + 3) * n));
    double* V = s.work64.p;
    GmCoop P{};
    P.n = n;
    P.m = m;
    P.maxiter = maxiter;
    P.tol = tol;
    P.dinv = s.dinv64.p;
    P.x = s.X.p;
    P.b = s.F.p;
    double out[5];
    MSFEM_TRY(gm_coop_run<double>(s, P, V, V + (size_t)(m + 1) * n, V + (size_t)(m + 2) * n, out));
    // the caller's residual report reads (F, F)
    MSFEM_CK(cudaMemcpyAsync(&s.kstate.p->ff, &out[4], sizeof(double), cudaMemcpyHostToDevice, s.stream));
    MSFEM_CK(cudaStreamSynchronize(s.stream));
    *iters = (int)out[0];
    *restarts = (int)out[1];
    return out[2] <= tol * tol * out[4] ? MSFEM_OK : MSFEM_NOT_CONVERGED;
}

// Inner solve of FP32 iterative refinement: GMRES(m) on the FP32 copy of the Jacobi-scaled matrix
// (unit diagonal, so no preconditioner), A d = b from d = 0, to ||b - A d|| <= tau ||b||.  The
// Krylov basis is FP32 (half the bytes of the FP64 solver per Arnoldi pass); the Hessenberg
// matrix, the rotations and every inner product are FP64.  V is (m+1) n floats, g two more n.
int gmres32_inner(System& s, int m, float* d, const float* b, float* V, float* g, int maxiter, double tau, int* iters)
{
    GmCoop P{};
    P.n = s.n_rows;
    P.m = m;
    P.maxiter = maxiter;
    P.tol = tau;
    P.x = d;
    P.b = b;
    P.zero_start = 1;
    double out[5];
    MSFEM_TRY(gm_coop_run<float>(s, P, V, g, g + s.n_rows, out));
    *iters = (int)out[0];
    return MSFEM_OK;
}

}  // namespace msfem
