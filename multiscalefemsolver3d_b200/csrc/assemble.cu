// Deterministic element assembly into the node-level portrait, one warp per row.
//
// The reference computes every element matrix in an OpenMP loop and then adds
// them into CSSD_Matrix serially, element by element, finding each target entry
// by a linear search of the row (FEM/FEM.h:1349-1384, CSSD_Matrix.h:307-363).
// Here a warp owns a node's row: its lanes form the geometry of the node's
// elements (one each), then every lane owns a row entry and adds the
// contributions of the elements that hold its column, in ascending element
// order -- the reference's order, no atomics, one launch, the same bits on every run.
//
// What bounds it: the FP64 adds and the shuffles over a row's elements (24 in a Kuhn
// grid); each element's geometry is formed four times, once per node, which is less
// than the launches cost that it replaces: one per element colour (38 on a Kuhn grid),
// each writing 16 entries per element back to memory, after a colouring whose 39 rounds
// over all elements took nine tenths of the time to build a system.  Assembly at 20^3 /
// 60^3 / 100^3, ms: elasticity 1.07 / 5.86 / 15.7 -> 0.055 / 0.70 / 3.1, scalar 0.42 / 0.63 / 2.3 ->
// 0.043 / 0.43 / 1.9; building the system 3.2 / 13.4 / 53 -> 0.33 / 1.4 / 5.6.
#include <cub/cub.cuh>

#include <algorithm>

#include "devutil.cuh"
#include "element.cuh"
#include "internal.cuh"

namespace msfem {
namespace {

enum RowKind { kScalar = 0, kScalar3 = 1, kElastic = 2, kTextbook = 3 };

struct RowMesh {
    int n_nodes;
    const int32_t* inc_ptr;
    const int32_t* inc_elem;
    const uint32_t* inc_slot;
    const int32_t* nrp;
    const int32_t* tets;
    const double* xyz;
    const int32_t* mat;
};

// kScalar (FEM_Grid.h:103-152, the one-point rule with weight V): A_IJ = V sigma g_I.g_J.
// kScalar3 (FEM_Grid.h:25-102, three coefficients at the centroid): A_IJ = V (S g_I.g_J + M / 16),
// F_I += V f / 4.
// kElastic (FEM_Grid.h:2125-2192): the reference forms B_J^T D B_I (3x6 * 6x6 * 6x3) at each of the 4
// quadrature points; for the isotropic D of Domain.h:53-78 with lambda = k*a and mu = k*b that product
// is, entry by entry,
//   A[I][J][a][b] = V * (lambda * gJ_a * gI_b + mu * gI_a * gJ_b + mu * delta_ab * gI.gJ)
// (g = basis gradient), which also equals the reference's mirrored blocks A[J][I] = A[I][J]^T, so all
// 16 blocks come from this one expression.
// kTextbook: the textbook orientation lambda gI_a gJ_b + mu gJ_a gI_b (the transpose of every block),
// symmetric positive semi-definite; used to build preconditioners, not by the reference.
// c0, c1, c2: kScalar sigma per material; kScalar3 S, M, f per element; elasticity lambda, mu per
// material ([n_mat][2]).
template <int KIND>
__global__ void __launch_bounds__(128) k_assemble_rows(RowMesh G, const double* __restrict__ c0,
                                                       const double* __restrict__ c1, const double* __restrict__ c2,
                                                       int n_mat, double* __restrict__ val, double* __restrict__ F,
                                                       int* __restrict__ bad)
{
    constexpr bool EL = KIND == kElastic || KIND == kTextbook;
    constexpr int NQ = EL ? 15 : 5;  // per element: gradients, lambda, mu, V / the four entries, the load
    constexpr int W = EL ? 9 : 1;
    __shared__ double sh[4][NQ * 32];
    const int lane = threadIdx.x & 31;
    double* q = sh[threadIdx.x >> 5];
    const int nw = gridDim.x * 4;
    for (int node = blockIdx.x * 4 + (threadIdx.x >> 5); node < G.n_nodes; node += nw) {
        const int b = G.inc_ptr[node], deg = G.inc_ptr[node + 1] - b;
        const int row = G.nrp[node], len = G.nrp[node + 1] - row;
        for (int s0 = 0; s0 < len || s0 == 0; s0 += 32) {  // 32 entries of the row at a time
            double acc[W];
#pragma unroll
            for (int k = 0; k < W; k++) acc[k] = 0.0;
            double load = 0.0;
            for (int e0 = 0; e0 < deg; e0 += 32) {
                uint32_t slots = 0xffffffffu;  // no entry: the row is shorter than 255
                int own = 0;
                if (e0 + lane < deg) {
                    const int e = G.inc_elem[b + e0 + lane];
                    const int m = KIND == kScalar3 ? 0 : (G.mat ? G.mat[e] : 0);
                    const bool known = KIND == kScalar3 || (m >= 0 && m < n_mat);
                    if (!known) atomicExch(bad, 1);
                    double lam = 0.0, mu = 0.0;
                    if (EL && known) {
                        lam = c0[2 * m];
                        mu = c0[2 * m + 1];
                    }
                    // E <= 0: the element contributes nothing (FEM/FEM.h:1355-1363)
                    if (known && (!EL || lam != 0.0 || mu != 0.0)) {
                        const int4 t = __ldg(reinterpret_cast<const int4*>(G.tets) + e);
                        const int v[4] = {t.x, t.y, t.z, t.w};
                        own = node == v[0] ? 0 : node == v[1] ? 1 : node == v[2] ? 2 : 3;
                        slots = G.inc_slot[b + e0 + lane];
                        TetGeom T;
                        tet_geometry(G.xyz, v, T);
                        if constexpr (EL) {
#pragma unroll
                            for (int J = 0; J < 4; J++)
#pragma unroll
                                for (int a = 0; a < 3; a++) q[(3 * J + a) * 32 + lane] = T.g[J][a];
                            q[12 * 32 + lane] = lam;
                            q[13 * 32 + lane] = mu;
                            q[14 * 32 + lane] = T.vol;
                        } else {
                            double gi[3];
#pragma unroll
                            for (int a = 0; a < 3; a++)
                                gi[a] = own == 0 ? T.g[0][a] : own == 1 ? T.g[1][a] : own == 2 ? T.g[2][a] : T.g[3][a];
                            const double k0 = KIND == kScalar ? c0[m] : c0[e], m16 = KIND == kScalar3 ? c1[e] / 16.0 : 0.0;
#pragma unroll
                            for (int J = 0; J < 4; J++) {
                                double k = k0 * (gi[0] * T.g[J][0] + gi[1] * T.g[J][1] + gi[2] * T.g[J][2]);
                                if (KIND == kScalar3) k += m16;
                                q[J * 32 + lane] = k * T.vol;
                            }
                            if (KIND == kScalar3) q[4 * 32 + lane] = c2[e] * T.vol / 4.0;
                        }
                    }
                }
                __syncwarp();
                const int n = min(32, deg - e0);
                for (int e = 0; e < n; e++) {
                    const uint32_t at = __shfl_sync(0xffffffffu, slots, e);
                    const int I = EL ? __shfl_sync(0xffffffffu, own, e) : 0;
                    if (KIND == kScalar3) load += q[4 * 32 + e];
                    if (at == 0xffffffffu) continue;
                    const uint32_t d = at ^ ((uint32_t)(s0 + lane) * 0x01010101u);
                    const int J = (d & 0xffu) == 0 ? 0 : (d & 0xff00u) == 0 ? 1 : (d & 0xff0000u) == 0 ? 2 : (d >> 24) == 0 ? 3 : -1;
                    if (J < 0) continue;
                    if constexpr (EL) {
                        double gi[3], gj[3];
#pragma unroll
                        for (int a = 0; a < 3; a++) {
                            gi[a] = q[(3 * I + a) * 32 + e];
                            gj[a] = q[(3 * J + a) * 32 + e];
                        }
                        const double lam = q[12 * 32 + e], mu = q[13 * 32 + e], V = q[14 * 32 + e];
                        const double dd = mu * (gi[0] * gj[0] + gi[1] * gj[1] + gi[2] * gj[2]);
#pragma unroll
                        for (int a = 0; a < 3; a++)
#pragma unroll
                            for (int c = 0; c < 3; c++) {
                                double k = KIND == kTextbook ? lam * gi[a] * gj[c] + mu * gj[a] * gi[c]
                                                             : lam * gj[a] * gi[c] + mu * gi[a] * gj[c];
                                if (a == c) k += dd;
                                acc[3 * a + c] += V * k;
                            }
                    } else {
                        acc[0] += q[J * 32 + e];
                    }
                }
                __syncwarp();
            }
            if (s0 + lane < len) {
                double* out = val + (int64_t)W * (row + s0 + lane);
#pragma unroll
                for (int k = 0; k < W; k++) out[k] += acc[k];
            }
            if (KIND == kScalar3 && s0 == 0 && lane == 0) F[node] += load;
        }
    }
}

template <int KIND>
int launch_rows(System& s, const double* c0, const double* c1, const double* c2, int n_mat, int* bad)
{
    const RowMesh G{s.n_nodes, s.inc_ptr.p, s.inc_elem.p, s.inc_slot.p, s.nrp.p, s.tets.p, s.xyz.p, s.mat.p};
    const int blocks = (int)std::min<int64_t>(((int64_t)s.n_nodes + 3) / 4, 148 * 64);
    k_assemble_rows<KIND><<<blocks, 128, 0, s.stream>>>(G, c0, c1, c2, n_mat, s.val.p, s.F.p, bad);
    MSFEM_CK(cudaGetLastError());
    s.total_launches += 1;
    return MSFEM_OK;
}

// ---- traction: per (face, vertex) contribution, then a per-node sum in face order
__global__ void k_traction_contrib(int n_faces, const int32_t* __restrict__ faces, const double* __restrict__ tr,
                                   const double* __restrict__ xyz, int n_nodes, int32_t* key, int32_t* idx,
                                   double* contrib, int* bad)
{
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_faces) return;
    int a = faces[3 * f], b = faces[3 * f + 1], c = faces[3 * f + 2];
    if (a < 0 || a >= n_nodes || b < 0 || b >= n_nodes || c < 0 || c >= n_nodes) {
        atomicExch(bad, 1);
        key[3 * f] = key[3 * f + 1] = key[3 * f + 2] = 0;
        idx[3 * f] = 3 * f;
        idx[3 * f + 1] = 3 * f + 1;
        idx[3 * f + 2] = 3 * f + 2;
        for (int q = 0; q < 9; q++) contrib[9 * f + q] = 0.0;
        return;
    }
    double u[3], w[3];
    for (int d = 0; d < 3; d++) {
        u[d] = xyz[3 * (int64_t)b + d] - xyz[3 * (int64_t)a + d];
        w[d] = xyz[3 * (int64_t)c + d] - xyz[3 * (int64_t)a + d];
    }
    double cr[3] = {u[1] * w[2] - u[2] * w[1], u[2] * w[0] - u[0] * w[2], u[0] * w[1] - u[1] * w[0]};
    double area = 0.5 * sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]);
    int nodes[3] = {a, b, c};
    for (int vtx = 0; vtx < 3; vtx++) {
        key[3 * f + vtx] = nodes[vtx];
        idx[3 * f + vtx] = 3 * f + vtx;
        for (int d = 0; d < 3; d++) contrib[3 * (3 * f + vtx) + d] = tr[3 * f + d] * area / 3.0;
    }
}

__global__ void k_traction_sum(int m, const int32_t* __restrict__ key, const int32_t* __restrict__ idx,
                               const double* __restrict__ contrib, double* F)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    if (i > 0 && key[i - 1] == key[i]) return;  // the first entry of each node's run adds the run
    const int node = key[i];
    double f0 = F[3 * (int64_t)node], f1 = F[3 * (int64_t)node + 1], f2 = F[3 * (int64_t)node + 2];
    for (int j = i; j < m && key[j] == node; j++) {
        const double* c = contrib + 3 * (int64_t)idx[j];
        f0 += c[0];
        f1 += c[1];
        f2 += c[2];
    }
    F[3 * (int64_t)node] = f0;
    F[3 * (int64_t)node + 1] = f1;
    F[3 * (int64_t)node + 2] = f2;
}

inline unsigned grid_for(int64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

int finish_assembly(System& s, DBuf<int>& bad)
{
    int h_bad = 0;
    MSFEM_CK(cudaMemcpyAsync(&h_bad, bad.p, sizeof(int), cudaMemcpyDeviceToHost, s.stream));
    MSFEM_CK(cudaEventRecord(s.ev1, s.stream));
    MSFEM_CK(cudaStreamSynchronize(s.stream));
    float ms = 0;
    cudaEventElapsedTime(&ms, s.ev0, s.ev1);
    s.stats.ms_assemble = ms;
    if (h_bad) {
        set_error("a material id is outside [0, n_materials)");
        return MSFEM_ERR_ARGUMENT;
    }
    s.invalidate_values();
    return MSFEM_OK;
}

}  // namespace

int assemble_scalar(System& s, const double* sigma, int n_mat)
{
    if (s.kind != MSFEM_SCALAR) {
        set_error("assemble_scalar on an elasticity system");
        return MSFEM_ERR_STATE;
    }
    if (n_mat <= 0 || !sigma) {
        set_error("assemble_scalar: no materials");
        return MSFEM_ERR_ARGUMENT;
    }
    DBuf<double>& d_sig = s.params;
    DBuf<int>& bad = s.flag;
    MSFEM_TRY(d_sig.alloc(n_mat));
    MSFEM_TRY(bad.alloc(8));
    MSFEM_CK(cudaEventRecord(s.ev0, s.stream));
    MSFEM_CK(cudaMemcpyAsync(d_sig.p, sigma, sizeof(double) * n_mat, cudaMemcpyHostToDevice, s.stream));
    MSFEM_CK(cudaMemsetAsync(bad.p, 0, sizeof(int), s.stream));
    MSFEM_TRY(launch_rows<kScalar>(s, d_sig.p, nullptr, nullptr, n_mat, bad.p));
    return finish_assembly(s, bad);
}

int assemble_scalar3(System& s, const double* S, const double* M, const double* f, bool on_device)
{
    if (s.kind != MSFEM_SCALAR) {
        set_error("assemble_scalar3 on an elasticity system");
        return MSFEM_ERR_STATE;
    }
    if (!S || !M || !f) {
        set_error("assemble_scalar3: coefficient arrays missing");
        return MSFEM_ERR_ARGUMENT;
    }
    const size_t ne = (size_t)s.n_tets;
    DBuf<double> coef;
    DBuf<int>& bad = s.flag;
    MSFEM_TRY(coef.alloc(3 * ne));
    MSFEM_TRY(bad.alloc(8));
    MSFEM_CK(cudaEventRecord(s.ev0, s.stream));
    const cudaMemcpyKind kind = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    MSFEM_CK(cudaMemcpyAsync(coef.p, S, sizeof(double) * ne, kind, s.stream));
    MSFEM_CK(cudaMemcpyAsync(coef.p + ne, M, sizeof(double) * ne, kind, s.stream));
    MSFEM_CK(cudaMemcpyAsync(coef.p + 2 * ne, f, sizeof(double) * ne, kind, s.stream));
    MSFEM_CK(cudaMemsetAsync(bad.p, 0, sizeof(int), s.stream));
    MSFEM_TRY(launch_rows<kScalar3>(s, coef.p, coef.p + ne, coef.p + 2 * ne, 0, bad.p));
    return finish_assembly(s, bad);
}

// Domain::forMech::SetIsotropic_D (Library/Domain.h:53-78): k = E(1-nu)/((1+nu)(1-2nu)),
// off-diagonal normal coupling a*k, shear b*k  ->  lambda = a*k, mu = b*k; E <= 0 gives a
// material that contributes nothing (FEM/FEM.h:1355-1363)
void lame_params(const double* E, const double* nu, int n_mat, double* lame)
{
    for (int m = 0; m < n_mat; m++) {
        if (E[m] <= 0) {
            lame[2 * m] = 0.0;
            lame[2 * m + 1] = 0.0;
            continue;
        }
        double k = E[m] * (1. - nu[m]) / (1. + nu[m]) / (1. - 2. * nu[m]);
        double b = (1. - 2. * nu[m]) / (2. * (1. - nu[m]));
        double a = nu[m] / (1. - nu[m]);
        lame[2 * m] = a * k;
        lame[2 * m + 1] = b * k;
    }
}

int assemble_elastic(System& s, const double* E, const double* nu, int n_mat, bool textbook)
{
    if (s.kind != MSFEM_ELASTIC) {
        set_error("assemble_elastic on a scalar system");
        return MSFEM_ERR_STATE;
    }
    if (n_mat <= 0 || !E || !nu) {
        set_error("assemble_elastic: no materials");
        return MSFEM_ERR_ARGUMENT;
    }
    std::vector<double> lame(2 * (size_t)n_mat);
    lame_params(E, nu, n_mat, lame.data());
    DBuf<double>& d_lame = s.params;
    DBuf<int>& bad = s.flag;
    MSFEM_TRY(d_lame.alloc(2 * (size_t)n_mat));
    MSFEM_TRY(bad.alloc(8));
    MSFEM_CK(cudaEventRecord(s.ev0, s.stream));
    MSFEM_CK(cudaMemcpyAsync(d_lame.p, lame.data(), sizeof(double) * 2 * n_mat, cudaMemcpyHostToDevice, s.stream));
    MSFEM_CK(cudaMemsetAsync(bad.p, 0, sizeof(int), s.stream));
    MSFEM_TRY((textbook ? launch_rows<kTextbook>(s, d_lame.p, nullptr, nullptr, n_mat, bad.p)
                        : launch_rows<kElastic>(s, d_lame.p, nullptr, nullptr, n_mat, bad.p)));
    // a matrix-free operator (kuhn.cu) can stand for the values only while they hold one assembly
    if (s.elastic_form == 0) {
        s.elastic_form = textbook ? 2 : 1;
        s.lame_host = lame;
    } else {
        s.elastic_form = -1;
    }
    return finish_assembly(s, bad);
}

int add_traction(System& s, int n_faces, const int32_t* d_faces, const double* d_traction)
{
    if (s.kind != MSFEM_ELASTIC) {
        set_error("add_traction needs an elasticity system");
        return MSFEM_ERR_STATE;
    }
    if (n_faces <= 0) return MSFEM_OK;
    const int m = 3 * n_faces;
    DBuf<int32_t>&key = s.sc_i32[1], &idx = s.sc_i32[2], &key2 = s.sc_i32[3], &idx2 = s.sc_i32[4];
    DBuf<double>& contrib = s.sc_f64[1];
    DBuf<int>& bad = s.flag;
    MSFEM_TRY(key.alloc(m));
    MSFEM_TRY(idx.alloc(m));
    MSFEM_TRY(key2.alloc(m));
    MSFEM_TRY(idx2.alloc(m));
    MSFEM_TRY(contrib.alloc(3 * (size_t)m));
    MSFEM_TRY(bad.alloc(8));
    MSFEM_CK(cudaMemsetAsync(bad.p, 0, sizeof(int), s.stream));
    k_traction_contrib<<<grid_for(n_faces, 128), 128, 0, s.stream>>>(n_faces, d_faces, d_traction, s.xyz.p, s.n_nodes,
                                                                     key.p, idx.p, contrib.p, bad.p);
    MSFEM_CK(cudaGetLastError());
    size_t tmp_bytes = 0;
    DBuf<unsigned char>& tmp = s.sc_tmp;
    cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, key.p, key2.p, idx.p, idx2.p, m, 0, 32, s.stream);
    MSFEM_TRY(tmp.alloc(tmp_bytes + 1));
    MSFEM_CK(cub::DeviceRadixSort::SortPairs(tmp.p, tmp_bytes, key.p, key2.p, idx.p, idx2.p, m, 0, 32, s.stream));
    k_traction_sum<<<grid_for(m, 128), 128, 0, s.stream>>>(m, key2.p, idx2.p, contrib.p, s.F.p);
    MSFEM_CK(cudaGetLastError());
    s.total_launches += 2;
    int h_bad = 0;
    MSFEM_CK(cudaMemcpyAsync(&h_bad, bad.p, sizeof(int), cudaMemcpyDeviceToHost, s.stream));
    MSFEM_CK(cudaStreamSynchronize(s.stream));
    if (h_bad) {
        set_error("a traction face references a node id outside [0, %d)", s.n_nodes);
        return MSFEM_ERR_ARGUMENT;
    }
    return MSFEM_OK;
}

}  // namespace msfem
