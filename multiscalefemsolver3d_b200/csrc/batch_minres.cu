// The persistent solver of the batched cell systems: one thread-block cluster per system.
//
// A cell problem has Dirichlet data on its whole boundary and zero source; its matrix is symmetric
// but, with stiff inclusions, indefinite (the reference's transposed element blocks leave interface
// terms; a few negative eigenvalues appear), so the inner solver is MINRES on the Jacobi-scaled free
// block S A_II S.  One persistent launch covers every system: each cluster takes the next system
// from an atomic queue (largest first), runs the FP64 outer refinement (true residual r = b - A x
// with the Dirichlet values in x) and the inner MINRES for all R right-hand sides at once (one
// recurrence per right-hand side, one shared sparse product).
//
// The free block is stored apart (BatchSys::scol / s64 / s32): free rows only, pre-scaled, in slices
// of G rows whose entries are interleaved, so that the G rows of a warp read one contiguous piece
// per matrix element.  A thread owns one row and two neighbouring right-hand sides (R = 4, 8), the
// work vectors are [row][component][right-hand side]: every access to them is a full 16-byte vector.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "batch.cuh"
#include "devutil.cuh"

namespace msfem {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxCluster = 16;

// A cluster of several CTAs a system; one CTA, whose barriers and sums are those of a block; one CTA whose system, of
// up to 8 slices and 128 rows (some 100 KB of FP64), stays in the L1.  Face problems, ms, with cluster barriers / of a
// block / and L1: 6 sheets of 8 squares per edge, FP32 to 1e-8, 0.39 / 0.33 / 0.27 (a CTA a system with a CSR product:
// 0.37), 3000 of them 5.5 / 2.5 / 2.0 (4.4); 12,000 of 5, FP64 to 1e-12, 8.0 / 3.1 / 2.4 (5.6).
enum Form { kCluster, kSolo, kTiny };

template <int R>
struct Lanes {
    static constexpr int NR = R >= 2 ? 2 : 1;  // right-hand sides per thread
    static constexpr int LPR = R / NR;         // lanes per row
    static constexpr int G = 32 / LPR;         // rows per warp and per slice
};

struct BatchArgs {
    int n_sys;
    const int32_t* order;
    const int64_t* node_off;
    const int64_t* row_ptr;
    const int32_t* col;
    const double* val64;
    const double* dscale;
    const int64_t* slice_off;   // [n_sys + 1] first slice of a system
    const int32_t* free_node;   // [n_slices * G] node of a free row, -1 past the system's last
    const int64_t* slice_ptr;   // [n_slices + 1] entries per row before the slice
    const int32_t* scol;
    const double* s64;
    const float* s32;
    double* x;
    const double* rhs;  // [n_nodes][R][3] source term, or null (zero source)
    void* work;
    int64_t work_stride;  // elements per vector
    int* queue;
    int32_t* iters;
    int32_t* outers;
    double* rel;
    double tol;
    int maxiter;
    int max_outer;
};

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ unsigned cluster_size()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

// all threads of the cluster; global and shared writes before it are visible after it
template <int FORM>
__device__ __forceinline__ void cluster_sync()
{
    if constexpr (FORM != kCluster) {
        __syncthreads();
        return;
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t remote_addr(const void* p, unsigned rank)
{
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

__device__ __forceinline__ void remote_store(double* p, unsigned rank, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote_addr(p, rank)), "d"(v) : "memory");
}

__device__ __forceinline__ void remote_store(int* p, unsigned rank, int v)
{
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(remote_addr(p, rank)), "r"(v) : "memory");
}

// matrix entries: read once per product, so they leave the L1 to the gathered vector; TINY systems fit it whole
template <bool TINY, class T>
__device__ __forceinline__ T load_entry(const T* p)
{
    if constexpr (TINY) {
        return __ldg(p);
    } else if constexpr (sizeof(T) == 8) {
        double v;
        asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
        return v;
    } else if constexpr (std::is_same_v<T, float>) {
        float v;
        asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
        return v;
    } else {
        int v;
        asm volatile("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
        return v;
    }
}

// NR neighbouring right-hand sides of one component
template <class T, int NR>
struct Pack;
template <>
struct Pack<double, 2> {
    double v[2];
    __device__ __forceinline__ void load(const double* p)
    {
        const double2 t = *reinterpret_cast<const double2*>(p);
        v[0] = t.x;
        v[1] = t.y;
    }
    __device__ __forceinline__ void store(double* p) const { *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]); }
};
template <>
struct Pack<float, 2> {
    float v[2];
    __device__ __forceinline__ void load(const float* p)
    {
        const float2 t = *reinterpret_cast<const float2*>(p);
        v[0] = t.x;
        v[1] = t.y;
    }
    __device__ __forceinline__ void store(float* p) const { *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]); }
};
template <class T>
struct Pack<T, 1> {
    T v[1];
    __device__ __forceinline__ void load(const T* p) { v[0] = *p; }
    __device__ __forceinline__ void store(T* p) const { *p = v[0]; }
};

struct MrRhs {
    double eta, c0, s0, c1, s1, eps, delta, ig, tau, b1, target, fnorm2;
    int active, upd;
};

// Shared state of one CTA (every CTA of the cluster holds the same scalars, computed from the same
// numbers in the same order).
template <int R>
struct CtaShared {
    double red[4][16 * R];             // partials per warp
    double slot[4][kMaxCluster * R];   // partials per CTA, written by every CTA of the cluster
    double s1[R], s2[R];
    MrRhs mr[R];
    double rr_prev[R];
    int s_bad[R];
    int q, conv, bad;
};

// One CTA's place in the cluster's system
template <int R, int FORM>
struct Place {
    int64_t slice0;        // first slice of the system
    int sl_lo, sl_hi;      // this CTA's slices within the system
    int warp, nw, lane, g, j;
    unsigned rank, size;
};

// sums a[] over the cluster for every right-hand side, in a fixed order: warp shuffles, the warps of
// a CTA, then the CTAs by rank.  One CTA barrier and one cluster barrier, which also makes the
// vectors written before it visible to the whole cluster.
//
// The slots are read after that barrier, so a buffer may be written again only when another cluster
// barrier has passed: two sums in a row never share one.  The residual takes buffers 2 and 3, the
// Krylov sums 0 and 1 in turn.
template <int R, int FORM, int N>
__device__ __forceinline__ void cluster_sum(CtaShared<R>& sh, const Place<R, FORM>& P, const int (&buf)[N],
                                            double (&a)[N][Lanes<R>::NR])
{
    using L = Lanes<R>;
#pragma unroll
    for (int q = 0; q < N; q++)
#pragma unroll
        for (int u = 0; u < L::NR; u++)
#pragma unroll
            for (int o = 16; o >= L::LPR; o >>= 1) a[q][u] += __shfl_xor_sync(kFull, a[q][u], o);
    if (P.lane < L::LPR)
#pragma unroll
        for (int q = 0; q < N; q++)
#pragma unroll
            for (int u = 0; u < L::NR; u++) sh.red[buf[q]][P.warp * R + P.lane * L::NR + u] = a[q][u];
    __syncthreads();
    if constexpr (FORM != kCluster) {  // the CTA's own sums, and no second barrier
#pragma unroll
        for (int q = 0; q < N; q++)
#pragma unroll
            for (int u = 0; u < L::NR; u++) {
                double s = 0.0;
                for (int w = 0; w < P.nw; w++) s += sh.red[buf[q]][w * R + P.j * L::NR + u];
                a[q][u] = s;
            }
        return;
    }
    for (int t = threadIdx.x; t < R * (int)P.size; t += blockDim.x) {
        const int r = t % R, dst = t / R;
#pragma unroll
        for (int q = 0; q < N; q++) {
            double s = 0.0;
            for (int w = 0; w < P.nw; w++) s += sh.red[buf[q]][w * R + r];
            remote_store(&sh.slot[buf[q]][P.rank * R + r], dst, s);
        }
    }
    cluster_sync<FORM>();
#pragma unroll
    for (int q = 0; q < N; q++)
#pragma unroll
        for (int u = 0; u < L::NR; u++) {
            double s = 0.0;
            for (unsigned c = 0; c < P.size; c++) s += sh.slot[buf[q]][c * R + P.j * L::NR + u];
            a[q][u] = s;
        }
}

// FP64 residual r = b - A x on the free rows (x holds the Dirichlet values), written scaled (S r)
// into V; ||r||^2 -> sh.s1, ||S r||^2 -> sh.s2 per right-hand side.
template <int R, class VT, int FORM>
__device__ void residual_pass(const BatchArgs& A, const Place<R, FORM>& P, VT* V, CtaShared<R>& sh)
{
    using L = Lanes<R>;
    double acc[2][L::NR] = {};
    const double* X = A.x;
    for (int sl = P.sl_lo + P.warp; sl < P.sl_hi; sl += P.nw) {
        const int row = sl * L::G + P.g;
        const int gi = A.free_node[P.slice0 * L::G + row];
        double y[3][L::NR] = {};
        if (gi < 0) {  // past the last row: zeros, which the products and sums below read
            Pack<VT, L::NR> z;
#pragma unroll
            for (int u = 0; u < L::NR; u++) z.v[u] = (VT)0;
#pragma unroll
            for (int c = 0; c < 3; c++) z.store(V + ((int64_t)row * 3 + c) * R + P.j * L::NR);
            continue;
        }
        if (A.rhs)
#pragma unroll
            for (int u = 0; u < L::NR; u++)
#pragma unroll
                for (int c = 0; c < 3; c++) y[c][u] = A.rhs[((int64_t)gi * R + P.j * L::NR + u) * 3 + c];
        for (int64_t k = A.row_ptr[gi]; k < A.row_ptr[gi + 1]; k++) {
            const double* a = A.val64 + 9 * k;
            const double* xv = X + ((int64_t)A.col[k] * R + P.j * L::NR) * 3;
#pragma unroll
            for (int u = 0; u < L::NR; u++)
#pragma unroll
                for (int c = 0; c < 3; c++)
                    y[c][u] -= a[3 * c] * xv[3 * u] + a[3 * c + 1] * xv[3 * u + 1] + a[3 * c + 2] * xv[3 * u + 2];
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double s = A.dscale[3 * (int64_t)gi + c];
            Pack<VT, L::NR> o;
#pragma unroll
            for (int u = 0; u < L::NR; u++) {
                acc[0][u] += y[c][u] * y[c][u];
                o.v[u] = (VT)(s * y[c][u]);
                acc[1][u] += (double)o.v[u] * (double)o.v[u];
            }
            o.store(V + ((int64_t)row * 3 + c) * R + P.j * L::NR);
        }
    }
    const int buf[2] = {2, 3};  // the first Krylov sum follows with no cluster barrier between
    cluster_sum(sh, P, buf, acc);
    if (threadIdx.x < L::LPR)
#pragma unroll
        for (int u = 0; u < L::NR; u++) {
            sh.s1[threadIdx.x * L::NR + u] = acc[0][u];
            sh.s2[threadIdx.x * L::NR + u] = acc[1][u];
        }
    __syncthreads();
}

// x += sign * S y on this CTA's free rows, for the right-hand sides with want[r] set (null: all)
template <int R, class VT, int FORM>
__device__ void apply_correction(const BatchArgs& A, const Place<R, FORM>& P, const VT* Y, double sign, const int* want)
{
    using L = Lanes<R>;
    for (int sl = P.sl_lo + P.warp; sl < P.sl_hi; sl += P.nw) {
        const int row = sl * L::G + P.g;
        const int gi = A.free_node[P.slice0 * L::G + row];
        if (gi < 0) continue;
#pragma unroll
        for (int u = 0; u < L::NR; u++) {
            const int r = P.j * L::NR + u;
            if (want && !want[r]) continue;
#pragma unroll
            for (int c = 0; c < 3; c++)
                A.x[((int64_t)gi * R + r) * 3 + c] +=
                    sign * A.dscale[3 * (int64_t)gi + c] * (double)Y[((int64_t)row * 3 + c) * R + r];
        }
    }
}

// MINRES on S A_II S y = u (U[0] on entry, ||u|| = mr[r].b1), all R right-hand sides at once; the
// solution is left in Y, the number of steps returned.
//
// The Lanczos vectors stay unnormalised (v_k = u_k / beta_k, the factor applied where u is read), so
// a step needs two cluster barriers: after q = A v_k with alpha = (v_k, q), and after
// u_{k+1} = q - alpha v_k - beta_k v_{k-1} with its norm.  The search direction and the solution of
// step k are updated during step k + 1, next to the pass that reads v_k anyway; the scalars of
// step k are formed by R threads while the others start the next product.
template <int R, class VT, int FORM>
__device__ int inner_minres(const BatchArgs& A, const Place<R, FORM>& P, const VT* __restrict__ mat, VT* base,
                            CtaShared<R>& sh)
{
    using L = Lanes<R>;
    using Pk = Pack<VT, L::NR>;
    const int64_t S = A.work_stride;
    VT* u_old = base;
    VT* u_cur = base + S;
    VT* u_new = base + 2 * S;
    VT* w2 = base + 3 * S;
    VT* w1 = base + 4 * S;
    VT* Y = base + 5 * S;
    const int jr = P.j * L::NR;
    for (int sl = P.sl_lo + P.warp; sl < P.sl_hi; sl += P.nw) {
        Pk z;
#pragma unroll
        for (int u = 0; u < L::NR; u++) z.v[u] = (VT)0;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const int64_t o = ((int64_t)(sl * L::G + P.g) * 3 + c) * R + jr;
            z.store(u_old + o);
            z.store(w1 + o);
            z.store(w2 + o);
            z.store(Y + o);
        }
    }
    VT ib[L::NR], ib_old[L::NR];
    double beta[L::NR];
#pragma unroll
    for (int u = 0; u < L::NR; u++) {
        const double b1 = sh.mr[jr + u].b1;
        ib[u] = (VT)(b1 > 0.0 ? 1.0 / b1 : 0.0);
        ib_old[u] = (VT)0;
        beta[u] = 0.0;
    }
    // w = (v - eps w2 - delta w1) / gamma into w2, y += tau w: the update of the step before
    auto direction = [&](int64_t o, const VT (&v)[L::NR], const bool (&on)[L::NR], const VT (&ep)[L::NR],
                         const VT (&de)[L::NR], const VT (&ig)[L::NR], const VT (&ta)[L::NR]) {
        Pk a, b, y;
        a.load(w2 + o);
        b.load(w1 + o);
        y.load(Y + o);
#pragma unroll
        for (int u = 0; u < L::NR; u++)
            if (on[u]) {  // a finished right-hand side keeps its solution
                a.v[u] = (v[u] - ep[u] * a.v[u] - de[u] * b.v[u]) * ig[u];
                y.v[u] += ta[u] * a.v[u];
            }
        a.store(w2 + o);
        y.store(Y + o);
    };
    int k = 0;
    for (;; k++) {
        // q = S A S v into u_new, alpha = (v, q)
        double a1[1][L::NR] = {};
        for (int sl = P.sl_lo + P.warp; sl < P.sl_hi; sl += P.nw) {
            const int64_t p0 = A.slice_ptr[P.slice0 + sl];
            const int width = (int)(A.slice_ptr[P.slice0 + sl + 1] - p0);
            const int32_t* cp = A.scol + p0 * L::G + P.g;
            const VT* mp = mat + p0 * 9 * L::G + P.g;
            VT acc[3][L::NR] = {};
#pragma unroll 3
            for (int e = 0; e < width; e++) {
                const int c = load_entry<FORM == kTiny>(cp + e * L::G);
                VT m[9];
#pragma unroll
                for (int t = 0; t < 9; t++) m[t] = load_entry<FORM == kTiny>(mp + (e * 9 + t) * L::G);
                const VT* xv = u_cur + (int64_t)c * 3 * R + jr;
                Pk x0, x1, x2;
                x0.load(xv);
                x1.load(xv + R);
                x2.load(xv + 2 * R);
#pragma unroll
                for (int t = 0; t < 3; t++)
#pragma unroll
                    for (int u = 0; u < L::NR; u++)
                        acc[t][u] += m[3 * t] * x0.v[u] + m[3 * t + 1] * x1.v[u] + m[3 * t + 2] * x2.v[u];
            }
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const int64_t o = ((int64_t)(sl * L::G + P.g) * 3 + c) * R + jr;
                Pk v, q;
                v.load(u_cur + o);
#pragma unroll
                for (int u = 0; u < L::NR; u++) {
                    q.v[u] = acc[c][u] * ib[u];
                    a1[0][u] += (double)(v.v[u] * ib[u]) * (double)q.v[u];
                }
                q.store(u_new + o);
            }
        }
        const int bufA[1] = {0};
        cluster_sum(sh, P, bufA, a1);
        // the scalars of step k - 1 are in place since the CTA barrier of the sum above
        if (k > 0) {
            int na = 0;
#pragma unroll
            for (int r = 0; r < R; r++) na |= sh.mr[r].active;
            if (na == 0) break;
        }
        if (k >= A.maxiter) break;
        VT al[L::NR], be[L::NR], ep[L::NR], de[L::NR], ig[L::NR], ta[L::NR];
        bool upd[L::NR];
        bool any = false;
#pragma unroll
        for (int u = 0; u < L::NR; u++) {
            const MrRhs& m = sh.mr[jr + u];
            al[u] = (VT)a1[0][u];
            be[u] = (VT)beta[u];
            upd[u] = k > 0 && m.upd;
            any |= upd[u];
            ep[u] = (VT)m.eps;
            de[u] = (VT)m.delta;
            ig[u] = (VT)m.ig;
            ta[u] = (VT)m.tau;
        }
        // u_new = q - alpha v - beta v_old and its norm; the direction and solution of step k - 1
        double a2[1][L::NR] = {};
        for (int sl = P.sl_lo + P.warp; sl < P.sl_hi; sl += P.nw)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const int64_t o = ((int64_t)(sl * L::G + P.g) * 3 + c) * R + jr;
                Pk q, v, vo;
                q.load(u_new + o);
                v.load(u_cur + o);
                vo.load(u_old + o);
                VT vold[L::NR];
#pragma unroll
                for (int u = 0; u < L::NR; u++) {
                    vold[u] = vo.v[u] * ib_old[u];
                    q.v[u] = q.v[u] - al[u] * (v.v[u] * ib[u]) - be[u] * vold[u];
                    a2[0][u] += (double)q.v[u] * (double)q.v[u];
                }
                q.store(u_new + o);
                if (any) direction(o, vold, upd, ep, de, ig, ta);
            }
        const int bufB[1] = {1};
        cluster_sum(sh, P, bufB, a2);
        double bn[L::NR];
#pragma unroll
        for (int u = 0; u < L::NR; u++) bn[u] = sqrt(a2[0][u]);
        if (threadIdx.x < R) {  // a right-hand side each: u of the NR whose sums this lane holds
            const bool second = L::NR == 2 && threadIdx.x >= L::LPR;
            const double al1 = second ? a1[0][L::NR - 1] : a1[0][0], b0 = second ? beta[L::NR - 1] : beta[0];
            const double b2 = second ? bn[L::NR - 1] : bn[0];
            MrRhs& m = sh.mr[jr + (second ? 1 : 0)];
            m.upd = m.active;
            if (m.active) {
                const double eps = m.s0 * b0;
                const double d1 = m.c0 * b0;
                const double delta = m.c1 * d1 + m.s1 * al1;
                const double g1 = -m.s1 * d1 + m.c1 * al1;
                const double gamma = sqrt(g1 * g1 + b2 * b2);
                const double inv = gamma > 0.0 ? 1.0 / gamma : 0.0;
                const double cs = gamma > 0.0 ? g1 / gamma : 1.0, sn = gamma > 0.0 ? b2 / gamma : 0.0;
                m.eps = eps;
                m.delta = delta;
                m.ig = inv;
                m.tau = gamma > 0.0 ? cs * m.eta : 0.0;
                m.eta = -sn * m.eta;
                m.c0 = m.c1;
                m.s0 = m.s1;
                m.c1 = cs;
                m.s1 = sn;
                if (!(gamma > 0.0) || !(b2 > 0.0) || fabs(m.eta) <= m.target * m.b1) m.active = 0;
                if (!(gamma > 0.0)) m.upd = 0;
            }
        }
#pragma unroll
        for (int u = 0; u < L::NR; u++) {
            beta[u] = bn[u];
            ib_old[u] = ib[u];
            ib[u] = (VT)(bn[u] > 0.0 ? 1.0 / bn[u] : 0.0);
        }
        VT* t = u_old;
        u_old = u_cur;
        u_cur = u_new;
        u_new = t;
        if (k > 0) {  // the direction written in this step is the newer one now
            t = w2;
            w2 = w1;
            w1 = t;
        }
    }
    // the last step's direction and solution
    if (k > 0) {
        VT ep[L::NR], de[L::NR], ig[L::NR], ta[L::NR];
        bool upd[L::NR];
#pragma unroll
        for (int u = 0; u < L::NR; u++) {
            const MrRhs& m = sh.mr[jr + u];
            upd[u] = m.upd;
            ep[u] = (VT)m.eps;
            de[u] = (VT)m.delta;
            ig[u] = (VT)m.ig;
            ta[u] = (VT)m.tau;
        }
        for (int sl = P.sl_lo + P.warp; sl < P.sl_hi; sl += P.nw)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const int64_t o = ((int64_t)(sl * L::G + P.g) * 3 + c) * R + jr;
                Pk vo;
                vo.load(u_old + o);
                VT v[L::NR];
#pragma unroll
                for (int u = 0; u < L::NR; u++) v[u] = vo.v[u] * ib_old[u];
                direction(o, v, upd, ep, de, ig, ta);
            }
    }
    return k;
}

// One cluster per system, taken from an atomic queue.  FP64 outer refinement; the inner solves start
// in FP32 (precision MSFEM_FP32_IR) and a system whose FP32 step fails to halve a right-hand side's
// residual has that step undone and continues with FP64 inner solves (ill-conditioned cells: FP32
// Lanczos vectors lose orthogonality).  Every CTA of the cluster takes the same decisions from the
// same numbers, so all reach the same barriers.
template <int R, int FORM>
__global__ void __launch_bounds__(512) k_batch_minres(BatchArgs A, int start64)
{
    using L = Lanes<R>;
    __shared__ CtaShared<R> sh;
    const int tid = threadIdx.x;
    Place<R, FORM> P;
    P.rank = cluster_rank();
    P.size = cluster_size();
    P.warp = tid >> 5;
    P.nw = blockDim.x >> 5;
    P.lane = tid & 31;
    P.g = P.lane / L::LPR;
    P.j = P.lane % L::LPR;
    char* base = reinterpret_cast<char*>(A.work) + (int64_t)(blockIdx.x / P.size) * 6 * A.work_stride * sizeof(double);
    float* base32 = reinterpret_cast<float*>(base);
    double* base64 = reinterpret_cast<double*>(base);
    cluster_sync<FORM>();  // every CTA runs before the first remote store

    for (;;) {
        if (P.rank == 0 && tid < (int)P.size) {
            int q = 0;
            if (tid == 0) q = atomicAdd(A.queue, 1);
            q = __shfl_sync((1u << P.size) - 1u, q, 0);
            remote_store(&sh.q, tid, q);
        }
        cluster_sync<FORM>();
        const int q = sh.q;
        if (q >= A.n_sys) break;
        const int sys = A.order[q];
        P.slice0 = A.slice_off[sys];
        const int ns = (int)(A.slice_off[sys + 1] - P.slice0);
        P.sl_lo = (int)((int64_t)ns * P.rank / P.size);
        P.sl_hi = (int)((int64_t)ns * (P.rank + 1) / P.size);
        if (tid < R) {
            sh.mr[tid].fnorm2 = 0.0;
            sh.rr_prev[tid] = 0.0;
            sh.s_bad[tid] = 0;
        }
        int use64 = start64, last64 = start64;
        int inner_total = 0, outer = 0;
        double relmax = 0.0;
        for (outer = 0;; outer++) {
            if (use64) residual_pass<R, double>(A, P, base64 + A.work_stride, sh);
            else residual_pass<R, float>(A, P, base32 + A.work_stride, sh);
            if (tid == 0) {
                // a right-hand side whose last FP32 step did not halve its residual
                int bad = 0;
                if (outer > 0 && !last64)
                    for (int r = 0; r < R; r++) {
                        sh.s_bad[r] = (sh.s1[r] > 0.25 * sh.rr_prev[r] && sh.rr_prev[r] > 0.0) ? 1 : 0;
                        bad |= sh.s_bad[r];
                    }
                sh.bad = bad;
            }
            __syncthreads();
            if (sh.bad) {
                // undo those steps (their corrections are still in Y) and recompute in FP64
                apply_correction<R, float>(A, P, base32 + 5 * A.work_stride, -1.0, sh.s_bad);
                cluster_sync<FORM>();
                use64 = 1;
                last64 = 1;
                if (tid < R) sh.s_bad[tid] = 0;
                residual_pass<R, double>(A, P, base64 + A.work_stride, sh);
            }
            if (tid == 0) {
                int conv = 1;
                double rm = 0.0;
                for (int r = 0; r < R; r++) {
                    if (outer == 0) sh.mr[r].fnorm2 = sh.s1[r];
                    const double rel = sh.mr[r].fnorm2 > 0.0 ? sqrt(sh.s1[r] / sh.mr[r].fnorm2) : 0.0;
                    rm = fmax(rm, rel);
                    const bool ok = rel <= A.tol;
                    conv &= ok ? 1 : 0;
                    sh.rr_prev[r] = sh.s1[r];
                    MrRhs& m = sh.mr[r];
                    m.b1 = sqrt(sh.s2[r]);
                    m.eta = m.b1;
                    m.c0 = m.c1 = 1.0;
                    m.s0 = m.s1 = 0.0;
                    // inner target: FP32 stops near its own precision, FP64 aims past the goal
                    const double need = rel > 0.0 ? A.tol / rel : 1.0;
                    m.target = use64 ? fmax(1e-15, 0.1 * need) : fmax(1e-5, fmin(0.5, 0.3 * need));
                    m.active = (!ok && m.b1 > 0.0) ? 1 : 0;
                    m.upd = 0;
                }
                sh.s1[0] = rm;
                sh.conv = conv || outer >= A.max_outer;
            }
            __syncthreads();
            relmax = sh.s1[0];
            if (sh.conv) break;
            if (use64) {
                inner_total += inner_minres<R, double>(A, P, A.s64, base64, sh);
                apply_correction<R, double>(A, P, base64 + 5 * A.work_stride, 1.0, nullptr);
            } else {
                inner_total += inner_minres<R, float>(A, P, A.s32, base32, sh);
                apply_correction<R, float>(A, P, base32 + 5 * A.work_stride, 1.0, nullptr);
            }
            last64 = use64;
            cluster_sync<FORM>();
        }
        if (P.rank == 0 && tid == 0) {
            A.iters[sys] = inner_total;
            A.outers[sys] = outer;
            A.rel[sys] = relmax;
        }
        cluster_sync<FORM>();  // sh.q and the scalars are free again
    }
}

// ------------------------------------------------------------------ the free block

__global__ void k_free_flags(int64_t n, const uint8_t* __restrict__ fixed, int32_t* __restrict__ flag)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += (int64_t)gridDim.x * blockDim.x)
        flag[i] = i < n && !fixed[i] ? 1 : 0;
}

// free rows before each system
__global__ void k_free_counts(int n_sys, const int64_t* __restrict__ node_off, const int32_t* __restrict__ pos,
                              int32_t* __restrict__ before)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s <= n_sys; s += gridDim.x * blockDim.x)
        before[s] = pos[node_off[s]];
}

// the free rows of a system, in node order, from its first slice on; lid: a node's row within its
// system, -1 for Dirichlet nodes
__global__ void k_free_rows(const int64_t* __restrict__ node_off, const int64_t* __restrict__ slice_off, int G,
                            const uint8_t* __restrict__ fixed, const int32_t* __restrict__ pos,
                            int32_t* __restrict__ free_node, int32_t* __restrict__ lid)
{
    const int s = blockIdx.x;
    const int64_t n0 = node_off[s];
    const int32_t before = pos[n0];
    for (int64_t i = n0 + threadIdx.x; i < node_off[s + 1]; i += blockDim.x) {
        const int l = fixed[i] ? -1 : pos[i] - before;
        lid[i] = l;
        if (l >= 0) free_node[slice_off[s] * G + l] = (int32_t)i;
    }
}

__global__ void k_slice_widths(int64_t n_rows, int G, const int32_t* __restrict__ free_node,
                               const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
                               const int32_t* __restrict__ lid, int* __restrict__ width)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_rows; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = free_node[t];
        if (i < 0) continue;
        int c = 0;
        for (int64_t k = row_ptr[i]; k < row_ptr[i + 1]; k++) c += lid[col[k]] >= 0;
        atomicMax(&width[t / G], c);
    }
}

// columns (PATTERN) or scaled values of the free block, row by row; shorter rows end in zero blocks
template <class T, bool PATTERN>
__global__ void k_fill_slices(int64_t n_rows, int G, const int32_t* __restrict__ free_node,
                              const int64_t* __restrict__ slice_ptr, const int64_t* __restrict__ row_ptr,
                              const int32_t* __restrict__ col, const int32_t* __restrict__ lid,
                              const double* __restrict__ val, const double* __restrict__ dscale,
                              int32_t* __restrict__ scol, T* __restrict__ out)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_rows; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = free_node[t], s = t / G, g = t % G;
        int64_t p = slice_ptr[s];
        const int64_t end = slice_ptr[s + 1];
        if (i >= 0) {
            double si[3];
            if (!PATTERN)
                for (int a = 0; a < 3; a++) si[a] = dscale[3 * i + a];
            for (int64_t k = row_ptr[i]; k < row_ptr[i + 1]; k++) {
                const int64_t j = col[k];
                if (lid[j] < 0) continue;
                if (PATTERN) {
                    scol[p * G + g] = lid[j];
                } else {
                    const double sj[3] = {dscale[3 * j], dscale[3 * j + 1], dscale[3 * j + 2]};
#pragma unroll
                    for (int a = 0; a < 3; a++)
#pragma unroll
                        for (int b = 0; b < 3; b++)
                            out[(p * 9 + 3 * a + b) * G + g] = (T)(si[a] * val[9 * k + 3 * a + b] * sj[b]);
                }
                p++;
            }
        }
        for (; p < end; p++) {
            if (PATTERN) {
                scol[p * G + g] = 0;
            } else {
                for (int e = 0; e < 9; e++) out[(p * 9 + e) * G + g] = (T)0;
            }
        }
    }
}

int rows_per_slice(int R) { return R == 8 ? Lanes<8>::G : R == 4 ? Lanes<4>::G : Lanes<1>::G; }

unsigned blocks_of(int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 16)); }

// the scaled values of the free block in the precision asked for, when the values changed since
template <class T>
int fill_values(BatchSys& b, DBuf<T>& out, bool& ok)
{
    if (ok) return 0;
    const int G = rows_per_slice(b.R);
    MSFEM_TRY(out.alloc(std::max<int64_t>(1, 9 * b.n_entries * G)));
    const int64_t rows = b.n_slices * G;
    if (rows)
        k_fill_slices<T, false><<<blocks_of(rows), 256, 0, b.stream>>>(rows, G, b.free_node.p, b.slice_ptr.p, b.row_ptr.p,
                                                                       b.col.p, b.lid.p, b.val64.p, b.dscale.p, nullptr,
                                                                       out.p);
    MSFEM_CK(cudaGetLastError());
    ok = true;
    return 0;
}

// The launch shape: CTAs per system (the cluster) and threads per CTA.  A product offers one slice per warp, so a
// cluster never has more warps than the largest system has slices, rounded up, and a system of a few slices no more
// than four.  Below that the cluster doubles while all systems together ask for at most 4 CTAs per SM (asked, not
// resident: 512 threads of 128 registers fill an SM alone): few systems are bound by the latency of one SM's share,
// many by what streams from L2 and HBM, where wider clusters only add barriers.  Measured (volume problems, 512
// threads, ms for clusters of 1 / 2 / 4 / 8 / 16), FP64 to 1e-12: 8 cells of 8..20 hexahedra per edge 157 / 81 / 45 /
// 23 / 14; 64 cells of 8..17: 106 / 56 / 31 / 26 / 33; 74 of 16: 97 / 57 / 61 / 57 / 65; 220 of 16: 184 / 157 / 161 /
// 165 / 191; 512 of 8..20: 322 / 303 / 339 / 380 / 427; FP32 refinement to 1e-8: 103 / 52 / 29 / 15 / 9; 75 / 38 / 20 /
// 14 / 19; 70 / 37 / 30 / 32 / 36; 115 / 90 / 81 / 94 / 108; 260 / 179 / 170 / 189 / 242.  So the rule is within a few
// percent of the best but for more than 130 cells of unequal sizes, which would gain from wider clusters (150 of 8..20:
// 147 with its 2, 118 with 4; 300: 292 with its 1, 199 with 2).  Face problems, six a cell, are fastest with its 1 or
// 2.  The one-CTA kernel with a CSR product that this replaced took 660 / 590 ms on the first two, and 12.6 ms against
// 0.9 on one cell of 8.  256 threads instead of 512 cost 1.2 to 1.7 times as much on many large systems, and are as
// fast where a system has fewer than 64 slices; warps without a slice cost their barriers (12,000 sheets of 16 free
// rows, FP64: 32 threads 2.4 ms, 128 5.3).
struct Shape {
    int threads, cluster;
};

Shape launch_shape(const BatchSys& b, int threads, int sms)
{
    if (threads <= 0)
        threads = b.max_slices <= 8 ? 32 * std::min(std::max(b.max_slices, 1), 4) : (b.max_slices < 64 ? 256 : 512);
    Shape s{threads, 1};
    while (s.cluster < kMaxCluster && s.cluster * (threads / 32) < b.max_slices &&
           (int64_t)b.n_sys * 2 * s.cluster <= 4 * (int64_t)sms)
        s.cluster *= 2;
    return s;
}

template <int R>
int launch_minres(BatchSys& b, double* d_x, int start64, double tol, int maxiter, const Shape& shape)
{
    const bool tiny = b.max_slices <= 8 && b.max_slices * Lanes<R>::G <= 128;
    auto kern = shape.cluster > 1 ? k_batch_minres<R, kCluster>
                : tiny            ? k_batch_minres<R, kTiny>
                                  : k_batch_minres<R, kSolo>;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = shape.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.blockDim = dim3(shape.threads);
    cfg.gridDim = dim3(shape.cluster);
    cfg.stream = b.stream;
    if (shape.cluster > 8)
        MSFEM_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    int clusters = 0;
    MSFEM_CK(cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg));
    clusters = std::min(std::max(clusters, 1), b.n_sys);
    cfg.gridDim = dim3(clusters * shape.cluster);
    const int64_t stride = ((b.max_slices * (int64_t)Lanes<R>::G * R * 3) + 31) / 32 * 32;
    const size_t need = (size_t)clusters * 6 * stride * sizeof(double);  // room for FP64 vectors
    if (b.work.n < need) MSFEM_TRY(b.work.alloc(need));
    MSFEM_TRY(b.queue.alloc(1));
    MSFEM_CK(cudaMemsetAsync(b.queue.p, 0, sizeof(int), b.stream));
    BatchArgs a{};
    a.n_sys = b.n_sys;
    a.order = b.order.p;
    a.node_off = b.node_off.p;
    a.row_ptr = b.row_ptr.p;
    a.col = b.col.p;
    a.val64 = b.val64.p;
    a.dscale = b.dscale.p;
    a.slice_off = b.slice_off.p;
    a.free_node = b.free_node.p;
    a.slice_ptr = b.slice_ptr.p;
    a.scol = b.scol.p;
    a.s64 = b.s64.p;
    a.s32 = b.s32.p;
    a.x = d_x;
    a.work = b.work.p;
    a.work_stride = stride;
    a.queue = b.queue.p;
    a.iters = b.iters.p;
    a.outers = b.outers.p;
    a.rel = b.rel.p;
    a.rhs = b.rhs;
    a.tol = tol;
    a.maxiter = maxiter;
    a.max_outer = 30;
    MSFEM_CK(cudaLaunchKernelEx(&cfg, kern, a, start64));
    return 0;
}

}  // namespace

int batch_build_free(BatchSys& b)
{
    cudaStream_t st = b.stream;
    const int G = rows_per_slice(b.R);
    DBuf<int32_t> flag, pos, before;
    DBuf<unsigned char> tmp;
    MSFEM_TRY(flag.alloc(b.n_nodes + 1));
    MSFEM_TRY(pos.alloc(b.n_nodes + 1));
    MSFEM_TRY(before.alloc(b.n_sys + 1));
    MSFEM_TRY(b.lid.alloc(std::max<int64_t>(1, b.n_nodes)));
    k_free_flags<<<blocks_of(b.n_nodes + 1), 256, 0, st>>>(b.n_nodes, b.fixed.p, flag.p);
    size_t ts = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, ts, flag.p, pos.p, (int64_t)(b.n_nodes + 1), st);
    MSFEM_TRY(tmp.alloc(std::max<size_t>(ts, 1)));
    MSFEM_CK(cub::DeviceScan::ExclusiveSum(tmp.p, ts, flag.p, pos.p, (int64_t)(b.n_nodes + 1), st));
    k_free_counts<<<blocks_of(b.n_sys + 1), 256, 0, st>>>(b.n_sys, b.node_off.p, pos.p, before.p);
    std::vector<int32_t> h(b.n_sys + 1);
    MSFEM_CK(cudaMemcpyAsync(h.data(), before.p, sizeof(int32_t) * (b.n_sys + 1), cudaMemcpyDeviceToHost, st));
    MSFEM_CK(cudaStreamSynchronize(st));
    std::vector<int64_t> off(b.n_sys + 1, 0);
    b.max_slices = 0;
    for (int s = 0; s < b.n_sys; s++) {
        const int64_t n = (h[s + 1] - h[s] + G - 1) / G;
        off[s + 1] = off[s] + n;
        b.max_slices = std::max<int>(b.max_slices, (int)n);
    }
    b.n_slices = off[b.n_sys];
    const int64_t rows = b.n_slices * G;
    MSFEM_TRY(b.slice_off.alloc(b.n_sys + 1));
    MSFEM_CK(cudaMemcpyAsync(b.slice_off.p, off.data(), sizeof(int64_t) * (b.n_sys + 1), cudaMemcpyHostToDevice, st));
    MSFEM_TRY(b.free_node.alloc(std::max<int64_t>(1, rows)));
    MSFEM_CK(cudaMemsetAsync(b.free_node.p, 0xff, sizeof(int32_t) * std::max<int64_t>(1, rows), st));
    if (b.n_sys)
        k_free_rows<<<b.n_sys, 128, 0, st>>>(b.node_off.p, b.slice_off.p, G, b.fixed.p, pos.p, b.free_node.p, b.lid.p);
    DBuf<int> width;
    MSFEM_TRY(width.alloc(b.n_slices + 1));
    MSFEM_CK(cudaMemsetAsync(width.p, 0, sizeof(int) * (b.n_slices + 1), st));
    if (rows)
        k_slice_widths<<<blocks_of(rows), 256, 0, st>>>(rows, G, b.free_node.p, b.row_ptr.p, b.col.p, b.lid.p, width.p);
    MSFEM_TRY(b.slice_ptr.alloc(b.n_slices + 1));
    cub::DeviceScan::ExclusiveScan(nullptr, ts, width.p, b.slice_ptr.p, cuda::std::plus<int64_t>(), (int64_t)0,
                                   (int64_t)(b.n_slices + 1), st);
    MSFEM_TRY(tmp.alloc(std::max<size_t>(ts, 1)));
    MSFEM_CK(cub::DeviceScan::ExclusiveScan(tmp.p, ts, width.p, b.slice_ptr.p, cuda::std::plus<int64_t>(), (int64_t)0,
                                            (int64_t)(b.n_slices + 1), st));
    MSFEM_CK(cudaMemcpyAsync(&b.n_entries, b.slice_ptr.p + b.n_slices, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    MSFEM_CK(cudaStreamSynchronize(st));  // `off` is released here too
    MSFEM_TRY(b.scol.alloc(std::max<int64_t>(1, b.n_entries * G)));
    if (rows)
        k_fill_slices<double, true><<<blocks_of(rows), 256, 0, st>>>(rows, G, b.free_node.p, b.slice_ptr.p, b.row_ptr.p,
                                                                     b.col.p, b.lid.p, nullptr, nullptr, b.scol.p,
                                                                     (double*)nullptr);
    MSFEM_CK(cudaGetLastError());
    MSFEM_CK(cudaStreamSynchronize(st));
    return 0;
}

int batch_threads(const BatchSys& b, int threads)
{
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return launch_shape(b, threads, sms).threads;
}

int batch_solve(BatchSys& b, double* d_x, int precision, double tol, int maxiter, int threads)
{
    if (b.n_sys == 0) return 0;
    const int start64 = precision == MSFEM_FP32_IR ? 0 : 1;
    if (threads > 0 && (threads % 32 != 0 || threads > 512)) {
        set_error("batched solve: threads per system must be a multiple of 32, at most 512");
        return MSFEM_ERR_ARGUMENT;
    }
    if (b.R != 1 && b.R != 4 && b.R != 8) {
        set_error("batched solve: %d right-hand sides per system (1, 4 or 8 supported)", b.R);
        return MSFEM_ERR_ARGUMENT;
    }
    MSFEM_TRY(fill_values(b, b.s64, b.s64_ok));
    if (!start64) MSFEM_TRY(fill_values(b, b.s32, b.s32_ok));
    int dev = 0, sms = 0;
    MSFEM_CK(cudaGetDevice(&dev));
    MSFEM_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const Shape shape = launch_shape(b, threads, sms);
    b.threads = shape.threads;
    switch (b.R) {
    case 4: return launch_minres<4>(b, d_x, start64, tol, maxiter, shape);
    case 8: return launch_minres<8>(b, d_x, start64, tol, maxiter, shape);
    default: return launch_minres<1>(b, d_x, start64, tol, maxiter, shape);
    }
}

}  // namespace msfem
