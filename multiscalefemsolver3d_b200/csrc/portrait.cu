// Mesh topology on the GPU: node -> element incidence, the node-level portrait
// (the reference's CreationPortrait, FEM/FEM_Grid.h:665-716 and :3236-3287), and for
// every incidence the positions of the element's four nodes in the node's row,
// which the assembly (one warp per row, assemble.cu) gathers by.
#include <cub/cub.cuh>

#include <climits>

#include "devutil.cuh"
#include "internal.cuh"

namespace msfem {
namespace {

__global__ void k_count_incidence(int n_tets, const int32_t* __restrict__ tets, int n_nodes, int32_t* cnt,
                                  int* bad)
{
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)n_tets * 4) return;
    int v = tets[t];
    if (v < 0 || v >= n_nodes) {
        atomicExch(bad, 1);
        return;
    }
    atomicAdd(&cnt[v], 1);
}

__global__ void k_fill_incidence(int n_tets, const int32_t* __restrict__ tets, const int32_t* __restrict__ ptr,
                                 int32_t* cursor, int32_t* inc)
{
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)n_tets * 4) return;
    int v = tets[t];
    int pos = atomicAdd(&cursor[v], 1);
    inc[ptr[v] + pos] = (int32_t)(t >> 2);
}

// Sort each node's element list ascending (lists are short: 24 for an interior Kuhn node).
__global__ void k_sort_incidence(int n_nodes, const int32_t* __restrict__ ptr, int32_t* inc)
{
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n_nodes) return;
    int b = ptr[v], e = ptr[v + 1];
    for (int i = b + 1; i < e; i++) {
        int x = inc[i], j = i - 1;
        while (j >= b && inc[j] > x) {
            inc[j + 1] = inc[j];
            j--;
        }
        inc[j + 1] = x;
    }
}

// One warp per node row: gather the nodes of all incident elements (self
// included) into shared memory, bitonic-sort them, drop duplicates.  Pass 0
// stores the unique count, pass 1 writes the sorted columns and, per incidence,
// the row positions of the element's nodes in four bytes (a row has at most
// kMaxCandidates - kMaxCandidates / 4 + 1 < 255 entries).
template <int PASS>
__global__ void k_portrait_rows(int n_nodes, const int32_t* __restrict__ tets, const int32_t* __restrict__ inc_ptr,
                                const int32_t* __restrict__ inc, int32_t* count, const int32_t* __restrict__ rp,
                                int32_t* col, uint32_t* inc_slot, int* overflow)
{
    constexpr int WPB = 4;
    __shared__ int buf[WPB][kMaxCandidates];
    __shared__ int uniq[PASS ? WPB : 1][PASS ? kMaxCandidates : 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int row = blockIdx.x * WPB + w;
    if (row >= n_nodes) return;
    int* s = buf[w];
    const int b = inc_ptr[row], deg = inc_ptr[row + 1] - b;
    const int nc = 4 * deg;
    if (nc > kMaxCandidates) {
        if (lane == 0) atomicMax(overflow, nc);
        return;
    }
    int size = 32;
    while (size < nc) size <<= 1;
    for (int i = lane; i < size; i += 32) {
        int v = INT_MAX;
        if (i < nc) v = tets[4 * (int64_t)inc[b + (i >> 2)] + (i & 3)];
        s[i] = v;
    }
    __syncwarp();
    for (int k = 2; k <= size; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = lane; i < size; i += 32) {
                int ixj = i ^ j;
                if (ixj > i) {
                    bool asc = (i & k) == 0;
                    int a = s[i], c = s[ixj];
                    if ((a > c) == asc) {
                        s[i] = c;
                        s[ixj] = a;
                    }
                }
            }
            __syncwarp();
        }
    int total = 0;
    const int out0 = PASS ? rp[row] : 0;
    for (int base = 0; base < size; base += 32) {
        int i = base + lane;
        int v = s[i];
        bool keep = (v != INT_MAX) && (i == 0 || s[i - 1] != v);
        unsigned m = __ballot_sync(0xffffffffu, keep);
        if (PASS && keep) {
            const int at = total + __popc(m & ((1u << lane) - 1u));
            col[out0 + at] = v;
            uniq[w][at] = v;
        }
        total += __popc(m);
    }
    if (!PASS && lane == 0) count[row] = total;
    if (PASS) {
        __syncwarp();
        for (int i = lane; i < deg; i += 32) {
            const int4 t = reinterpret_cast<const int4*>(tets)[inc[b + i]];
            const int node[4] = {t.x, t.y, t.z, t.w};
            uint32_t packed = 0;
#pragma unroll
            for (int a = 0; a < 4; a++) {
                int lo = 0, hi = total - 1;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (uniq[w][mid] < node[a]) lo = mid + 1;
                    else hi = mid;
                }
                packed |= (uint32_t)lo << (8 * a);
            }
            inc_slot[b + i] = packed;
        }
    }
}

inline unsigned grid_for(int64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

}  // namespace

int build_topology(System& s)
{
    cudaStream_t st = s.stream;
    const int N = s.n_nodes, E = s.n_tets;
    DBuf<int> flags;  // [0] bad node id, [1] overflow
    MSFEM_TRY(flags.alloc(8));
    MSFEM_CK(cudaMemsetAsync(flags.p, 0, 8 * sizeof(int), st));

    // ---- incidence
    MSFEM_TRY(s.inc_ptr.alloc((size_t)N + 1));
    MSFEM_TRY(s.inc_elem.alloc((size_t)E * 4));
    DBuf<int32_t> cnt;
    MSFEM_TRY(cnt.alloc((size_t)N + 1));
    MSFEM_CK(cudaMemsetAsync(cnt.p, 0, sizeof(int32_t) * ((size_t)N + 1), st));
    k_count_incidence<<<grid_for((int64_t)E * 4, 256), 256, 0, st>>>(E, s.tets.p, N, cnt.p, flags.p);
    MSFEM_CK(cudaGetLastError());
    int h_flags[4];
    MSFEM_CK(cudaMemcpyAsync(h_flags, flags.p, sizeof(h_flags), cudaMemcpyDeviceToHost, st));
    MSFEM_CK(cudaStreamSynchronize(st));
    if (h_flags[0]) {  // checked before any kernel indexes by node id
        set_error("tets reference a node id outside [0, %d)", N);
        return MSFEM_ERR_ARGUMENT;
    }

    size_t tmp_bytes = 0;
    DBuf<unsigned char> tmp;
    cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, cnt.p, s.inc_ptr.p, N + 1, st);
    MSFEM_TRY(tmp.alloc(tmp_bytes + 1));
    MSFEM_CK(cub::DeviceScan::ExclusiveSum(tmp.p, tmp_bytes, cnt.p, s.inc_ptr.p, N + 1, st));
    MSFEM_CK(cudaMemsetAsync(cnt.p, 0, sizeof(int32_t) * ((size_t)N + 1), st));
    k_fill_incidence<<<grid_for((int64_t)E * 4, 256), 256, 0, st>>>(E, s.tets.p, s.inc_ptr.p, cnt.p, s.inc_elem.p);
    k_sort_incidence<<<grid_for(N, 128), 128, 0, st>>>(N, s.inc_ptr.p, s.inc_elem.p);
    MSFEM_CK(cudaGetLastError());

    // ---- node-level portrait
    MSFEM_TRY(s.nrp.alloc((size_t)N + 1));
    k_portrait_rows<0><<<grid_for(N, 4), 128, 0, st>>>(N, s.tets.p, s.inc_ptr.p, s.inc_elem.p, cnt.p, nullptr,
                                                       nullptr, nullptr, flags.p + 1);
    MSFEM_CK(cudaGetLastError());
    MSFEM_CK(cudaMemsetAsync(cnt.p + N, 0, sizeof(int32_t), st));
    tmp_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, cnt.p, s.nrp.p, N + 1, st);
    MSFEM_TRY(tmp.alloc(tmp_bytes + 1));
    MSFEM_CK(cub::DeviceScan::ExclusiveSum(tmp.p, tmp_bytes, cnt.p, s.nrp.p, N + 1, st));
    int32_t nnzb = 0;
    MSFEM_CK(cudaMemcpyAsync(&nnzb, s.nrp.p + N, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    MSFEM_CK(cudaMemcpyAsync(h_flags, flags.p, sizeof(h_flags), cudaMemcpyDeviceToHost, st));
    MSFEM_CK(cudaStreamSynchronize(st));
    if (h_flags[1]) {
        set_error("a node belongs to %d element-vertex slots; the portrait builder handles at most %d (node degree <= %d)",
                  h_flags[1], kMaxCandidates, kMaxCandidates / 4);
        return MSFEM_ERR_LIMIT;
    }
    s.nnzb = nnzb;
    MSFEM_TRY(s.ncol.alloc((size_t)nnzb));
    MSFEM_TRY(s.inc_slot.alloc((size_t)E * 4));
    k_portrait_rows<1><<<grid_for(N, 4), 128, 0, st>>>(N, s.tets.p, s.inc_ptr.p, s.inc_elem.p, nullptr, s.nrp.p,
                                                       s.ncol.p, s.inc_slot.p, flags.p + 1);
    MSFEM_CK(cudaGetLastError());
    MSFEM_CK(cudaStreamSynchronize(st));
    s.stats.n_colors = 1;  // the assembly is one launch over the rows
    // incidence count / fill / sort, portrait count / fill
    s.total_launches += 5;

    return MSFEM_OK;
}

}  // namespace msfem
