// Batched cell systems: sort-based deterministic portrait + assembly (the persistent solver is
// batch_minres.cu).
//
// Portrait and assembly.  The reference builds each cell problem's portrait
// (Grid_forMech::CreationPortrait, FEM/FEM_Grid.h:3236-3287) and adds the element
// matrices serially in element order (CSSD_Matrix::SummPartOfMatrix,
// Library/CSSD_Matrix.h:307-363), one cell at a time in an OpenMP loop over cells
// (MsFEM/MsFEM_Grid.h:4800-4802).  Here every element of every system emits its
// (k+1)^2 (row, column) node pairs, tagged element << 2b | I << b | J (b = 2 bits for up to 4
// nodes per element, 3 for 8); one stable
// radix sort by (row, column) groups equal pairs (a block of the matrix) with
// their contributions in element order.  The unique keys are the portrait (rows
// sorted, diagonal included); the sorted tags are kept, so assembling a block is
// a gather-sum of its contributions in the same order as the reference's serial
// scatter -- no colouring, no atomics, the same bits on every run.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <numeric>

#include "batch.cuh"
#include "devutil.cuh"
#include "element.cuh"

namespace msfem {
namespace {

constexpr unsigned kFull = 0xffffffffu;

int bits_for(int64_t n)
{
    int b = 1;
    while (((int64_t)1 << b) < n) b++;
    return b;
}

__global__ void k_check_elements(int n_sys, const int64_t* __restrict__ node_off, const int64_t* __restrict__ elem_off,
                                 const int32_t* __restrict__ elems, int k1, int* bad)
{
    const int s = blockIdx.x;
    if (s >= n_sys) return;
    const int64_t n0 = node_off[s], n1 = node_off[s + 1];
    for (int64_t e = elem_off[s] + threadIdx.x; e < elem_off[s + 1]; e += blockDim.x)
        for (int a = 0; a < k1; a++) {
            const int64_t v = elems[e * k1 + a];
            if (v < n0 || v >= n1) atomicExch(bad, 1);
        }
}

// bits of each element-local index in a contribution tag (element << 2 tb | I << tb | J)
__host__ __device__ __forceinline__ int tag_bits(int k1) { return k1 > 8 ? 5 : (k1 > 4 ? 3 : 2); }

__global__ void k_emit_pairs(int64_t e0, int64_t e1, int64_t n0, int nb, const int32_t* __restrict__ elems, int k1,
                             uint64_t* __restrict__ key, uint32_t* __restrict__ tag)
{
    const int64_t kk = (int64_t)k1 * k1;
    const int64_t count = (e1 - e0) * kk;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = e0 + t / kk;
        const int ab = (int)(t % kk);
        const int a = ab / k1, b = ab % k1;
        const uint64_t row = (uint64_t)(elems[e * k1 + a] - n0);
        const uint64_t col = (uint64_t)(elems[e * k1 + b] - n0);
        key[t] = (row << nb) | col;
        const int tb = tag_bits(k1);
        tag[t] = ((uint32_t)e << (2 * tb)) | (uint32_t)(a << tb) | (uint32_t)b;
    }
}

__global__ void k_heads(int64_t count, const uint64_t* __restrict__ key, int32_t* __restrict__ head)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
        head[i] = (i == 0 || key[i] != key[i - 1]) ? 1 : 0;
}

// one thread per sorted pair that starts a block: its column, first contribution, row count
__global__ void k_slots(int64_t count, const uint64_t* __restrict__ key, const int32_t* __restrict__ head,
                        const int32_t* __restrict__ slot, int64_t n0, int nb, int64_t pair_base,
                        int32_t* __restrict__ col, int64_t* __restrict__ cstart, int32_t* __restrict__ row_cnt)
{
    const uint64_t mask = ((uint64_t)1 << nb) - 1;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        if (!head[i]) continue;
        const int s = slot[i];
        const uint64_t k = key[i];
        col[s] = (int32_t)(n0 + (int64_t)(k & mask));
        cstart[s] = pair_base + i;
        atomicAdd(&row_cnt[n0 + (int64_t)(k >> nb)], 1);
    }
}

template <int K1>
__device__ __forceinline__ void element_block_of(const int32_t* __restrict__ elems, const double* __restrict__ xyz,
                                                 int64_t e, int I, int J, double lam, double mu, double out[9])
{
    if (K1 == 4) {
        int v[4];
#pragma unroll
        for (int a = 0; a < 4; a++) v[a] = elems[e * 4 + a];
        TetGeom G;
        tet_geometry(xyz, v, G);
        elastic_block(G.g[I], G.g[J], G.vol, lam, mu, out);
    } else {
        int v[3];
#pragma unroll
        for (int a = 0; a < 3; a++) v[a] = elems[e * 3 + a];
        double g[3][3], area;
        tri_geometry(xyz, v, g, area);
        elastic_block(g[I], g[J], area, lam, mu, out);
    }
}

// each block = sum of its element contributions in element order
template <int K1>
__global__ void k_assemble_blocks(int64_t nnzb, const int64_t* __restrict__ cstart, const uint32_t* __restrict__ contrib,
                                  const int32_t* __restrict__ elems, const int32_t* __restrict__ emat,
                                  const double* __restrict__ xyz, const double* __restrict__ lame, int n_mat,
                                  double* __restrict__ val, int* bad)
{
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < nnzb; s += (int64_t)gridDim.x * blockDim.x) {
        double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int64_t c = cstart[s]; c < cstart[s + 1]; c++) {
            const uint32_t t = contrib[c];
            const int64_t e = t >> 4;
            const int I = (t >> 2) & 3, J = t & 3;
            const int m = emat ? emat[e] : 0;
            if (m < 0 || m >= n_mat) {
                atomicExch(bad, 1);
                continue;
            }
            const double lam = lame[2 * m], mu = lame[2 * m + 1];
            if (lam == 0.0 && mu == 0.0) continue;  // E <= 0: no contribution (FEM/FEM.h:1355-1363)
            double blk[9];
            element_block_of<K1>(elems, xyz, e, I, J, lam, mu, blk);
#pragma unroll
            for (int q = 0; q < 9; q++) acc[q] += blk[q];
        }
#pragma unroll
        for (int q = 0; q < 9; q++) val[9 * s + q] = acc[q];
    }
}

// each block = sum of the caller's element blocks eb[e][I][J][9] in element order (8-node
// elements: the MsFEM macro cells)
__global__ void k_assemble_given(int64_t nnzb, const int64_t* __restrict__ cstart, const uint32_t* __restrict__ contrib,
                                 int k1, const double* __restrict__ eb, double* __restrict__ val)
{
    const int tb = tag_bits(k1);
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < nnzb; s += (int64_t)gridDim.x * blockDim.x) {
        double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int64_t c = cstart[s]; c < cstart[s + 1]; c++) {
            const uint32_t t = contrib[c];
            const int64_t e = t >> (2 * tb);
            const int I = (t >> tb) & ((1 << tb) - 1), J = t & ((1 << tb) - 1);
            const double* blk = eb + 9 * (((int64_t)e * k1 + I) * k1 + J);
#pragma unroll
            for (int q = 0; q < 9; q++) acc[q] += blk[q];
        }
#pragma unroll
        for (int q = 0; q < 9; q++) val[9 * s + q] = acc[q];
    }
}

// s = 1/sqrt(A_ii[a][a]) (1 when not positive)
__global__ void k_batch_scale(int64_t n_nodes, const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
                              const double* __restrict__ val, double* __restrict__ dscale)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_nodes; i += (int64_t)gridDim.x * blockDim.x) {
        double d[3] = {0, 0, 0};
        for (int64_t k = row_ptr[i]; k < row_ptr[i + 1]; k++)
            if (col[k] == i) {
                d[0] = val[9 * k];
                d[1] = val[9 * k + 4];
                d[2] = val[9 * k + 8];
            }
        for (int a = 0; a < 3; a++) dscale[3 * i + a] = d[a] > 0.0 ? 1.0 / sqrt(d[a]) : 1.0;
    }
}

}  // namespace

int batch_build_pattern(BatchSys& b, const double* d_xyz)
{
    (void)d_xyz;
    cudaStream_t st = b.stream;
    if (b.k1 > 32 || b.n_elems >= ((int64_t)1 << (32 - 2 * tag_bits(b.k1)))) {
        set_error("batched systems: %lld elements of %d nodes exceed the contribution tags", (long long)b.n_elems, b.k1);
        return MSFEM_ERR_LIMIT;
    }
    if (b.n_nodes >= ((int64_t)1 << 31)) {
        set_error("batched systems: node count exceeds the int32 range");
        return MSFEM_ERR_LIMIT;
    }
    // element nodes inside their own system
    DBuf<int> flag;
    MSFEM_TRY(flag.alloc(1));
    MSFEM_CK(cudaMemsetAsync(flag.p, 0, sizeof(int), st));
    if (b.n_sys > 0) k_check_elements<<<b.n_sys, 128, 0, st>>>(b.n_sys, b.node_off.p, b.elem_off.p, b.elems.p, b.k1, flag.p);
    int bad = 0;
    MSFEM_CK(cudaMemcpyAsync(&bad, flag.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    MSFEM_CK(cudaStreamSynchronize(st));
    if (bad) {
        set_error("batched systems: an element references a node outside its system");
        return MSFEM_ERR_ARGUMENT;
    }
    b.max_nodes = 0;
    for (int s = 0; s < b.n_sys; s++) b.max_nodes = std::max<int>(b.max_nodes, (int)(b.h_node_off[s + 1] - b.h_node_off[s]));
    const int kk = b.k1 * b.k1;
    b.n_pairs = b.n_elems * kk;
    MSFEM_TRY(b.contrib.alloc(std::max<int64_t>(1, b.n_pairs)));
    DBuf<int32_t> row_cnt;
    MSFEM_TRY(row_cnt.alloc(b.n_nodes + 1));
    MSFEM_CK(cudaMemsetAsync(row_cnt.p, 0, sizeof(int32_t) * (b.n_nodes + 1), st));

    // chunks of whole systems, at most kChunkPairs pairs each
    const int64_t kChunkPairs = (int64_t)1 << 28;
    struct Chunk {
        int64_t nslots;
        DBuf<int32_t> col;
        DBuf<int64_t> cstart;
    };
    std::vector<Chunk*> chunks;
    DBuf<uint64_t> keys[2];
    DBuf<uint32_t> tags[2];
    DBuf<int32_t> head, slot;
    DBuf<unsigned char> tmp;
    int s0 = 0;
    int rc = 0;
    while (s0 < b.n_sys && rc == 0) {
        int s1 = s0 + 1;
        while (s1 < b.n_sys && (b.h_elem_off[s1 + 1] - b.h_elem_off[s0]) * kk <= kChunkPairs) s1++;
        const int64_t e0 = b.h_elem_off[s0], e1 = b.h_elem_off[s1];
        const int64_t n0 = b.h_node_off[s0], n1 = b.h_node_off[s1];
        const int64_t P = (e1 - e0) * kk;
        if (P >= ((int64_t)1 << 31)) {
            set_error("batched systems: one system has more than 2^31 element pairs");
            rc = MSFEM_ERR_LIMIT;
            break;
        }
        auto* ch = new Chunk();
        chunks.push_back(ch);
        if (P == 0) {
            ch->nslots = 0;
            s0 = s1;
            continue;
        }
        const int nb = bits_for(n1 - n0);
        if ((rc = keys[0].alloc(P)) || (rc = keys[1].alloc(P)) || (rc = tags[0].alloc(P)) || (rc = tags[1].alloc(P)) ||
            (rc = head.alloc(P)) || (rc = slot.alloc(P)))
            break;
        const int blocks = (int)std::min<int64_t>((P + 255) / 256, 148 * 16);
        k_emit_pairs<<<blocks, 256, 0, st>>>(e0, e1, n0, nb, b.elems.p, b.k1, keys[0].p, tags[0].p);
        cub::DoubleBuffer<uint64_t> dk(keys[0].p, keys[1].p);
        cub::DoubleBuffer<uint32_t> dv(tags[0].p, tags[1].p);
        size_t tb = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, tb, dk, dv, (int)P, 0, 2 * nb, st);
        if ((rc = tmp.alloc(std::max(tb, (size_t)1)))) break;
        MSFEM_CK(cub::DeviceRadixSort::SortPairs(tmp.p, tb, dk, dv, (int)P, 0, 2 * nb, st));
        k_heads<<<blocks, 256, 0, st>>>(P, dk.Current(), head.p);
        size_t ts = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, ts, head.p, slot.p, (int)P, st);
        if ((rc = tmp.alloc(std::max(ts, tb)))) break;
        MSFEM_CK(cub::DeviceScan::ExclusiveSum(tmp.p, ts, head.p, slot.p, (int)P, st));
        int last_slot = 0, last_head = 0;
        MSFEM_CK(cudaMemcpyAsync(&last_slot, slot.p + P - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
        MSFEM_CK(cudaMemcpyAsync(&last_head, head.p + P - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
        MSFEM_CK(cudaStreamSynchronize(st));
        ch->nslots = (int64_t)last_slot + last_head;
        if ((rc = ch->col.alloc(ch->nslots)) || (rc = ch->cstart.alloc(ch->nslots))) break;
        const int64_t pair_base = e0 * kk;
        k_slots<<<blocks, 256, 0, st>>>(P, dk.Current(), head.p, slot.p, n0, nb, pair_base, ch->col.p, ch->cstart.p,
                                        row_cnt.p);
        MSFEM_CK(cudaMemcpyAsync(b.contrib.p + pair_base, dv.Current(), sizeof(uint32_t) * P, cudaMemcpyDeviceToDevice, st));
        MSFEM_CK(cudaGetLastError());
        s0 = s1;
    }
    if (rc == 0) {
        int64_t total = 0;
        for (auto* ch : chunks) total += ch->nslots;
        b.nnzb = total;
        if (!(rc = b.col.alloc(std::max<int64_t>(1, total))) && !(rc = b.cstart.alloc(total + 1)) &&
            !(rc = b.row_ptr.alloc(b.n_nodes + 1))) {
            int64_t off = 0;
            for (auto* ch : chunks) {
                if (ch->nslots) {
                    cudaMemcpyAsync(b.col.p + off, ch->col.p, sizeof(int32_t) * ch->nslots, cudaMemcpyDeviceToDevice, st);
                    cudaMemcpyAsync(b.cstart.p + off, ch->cstart.p, sizeof(int64_t) * ch->nslots, cudaMemcpyDeviceToDevice, st);
                }
                off += ch->nslots;
            }
            const int64_t np = b.n_pairs;
            MSFEM_CK(cudaMemcpyAsync(b.cstart.p + total, &np, sizeof(int64_t), cudaMemcpyHostToDevice, st));
            // row_ptr = exclusive scan of the per-row block counts (64-bit)
            DBuf<int64_t> cnt64;
            if (!(rc = cnt64.alloc(b.n_nodes + 1))) {
                std::vector<int32_t> h(b.n_nodes);
                MSFEM_CK(cudaMemcpyAsync(h.data(), row_cnt.p, sizeof(int32_t) * b.n_nodes, cudaMemcpyDeviceToHost, st));
                MSFEM_CK(cudaStreamSynchronize(st));
                std::vector<int64_t> rp(b.n_nodes + 1, 0);
                for (int64_t i = 0; i < b.n_nodes; i++) rp[i + 1] = rp[i] + h[i];
                if (rp[b.n_nodes] != total) {
                    set_error("batched systems: row counts (%lld) disagree with the block count (%lld)",
                              (long long)rp[b.n_nodes], (long long)total);
                    rc = MSFEM_ERR_STATE;
                } else {
                    MSFEM_CK(cudaMemcpyAsync(b.row_ptr.p, rp.data(), sizeof(int64_t) * (b.n_nodes + 1),
                                             cudaMemcpyHostToDevice, st));
                    MSFEM_CK(cudaStreamSynchronize(st));
                }
            }
        }
    }
    MSFEM_CK(cudaStreamSynchronize(st));
    for (auto* ch : chunks) delete ch;
    if (rc) return rc;
    // largest systems first
    std::vector<int32_t> ord(b.n_sys);
    std::iota(ord.begin(), ord.end(), 0);
    std::stable_sort(ord.begin(), ord.end(), [&](int a, int c) {
        return b.h_node_off[a + 1] - b.h_node_off[a] > b.h_node_off[c + 1] - b.h_node_off[c];
    });
    MSFEM_TRY(b.order.alloc(std::max(1, b.n_sys)));
    if (b.n_sys) MSFEM_CK(cudaMemcpyAsync(b.order.p, ord.data(), sizeof(int32_t) * b.n_sys, cudaMemcpyHostToDevice, st));
    MSFEM_TRY(b.iters.alloc(std::max(1, b.n_sys)));
    MSFEM_TRY(b.outers.alloc(std::max(1, b.n_sys)));
    MSFEM_TRY(b.rel.alloc(std::max(1, b.n_sys)));
    MSFEM_CK(cudaStreamSynchronize(st));
    return b.fixed.p ? batch_build_free(b) : 0;
}

int batch_assemble_enqueue(BatchSys& b, const double* d_xyz, const double* d_lame, int n_mat)
{
    cudaStream_t st = b.stream;
    MSFEM_TRY(b.val64.alloc(std::max<int64_t>(1, 9 * b.nnzb)));
    MSFEM_TRY(b.dscale.alloc(std::max<int64_t>(1, 3 * b.n_nodes)));
    DBuf<int>& flag = b.aflag;
    MSFEM_TRY(flag.alloc(1));
    MSFEM_CK(cudaMemsetAsync(flag.p, 0, sizeof(int), st));
    const int blocks = (int)std::min<int64_t>((b.nnzb + 255) / 256, 148 * 16);
    if (b.nnzb) {
        if (b.k1 == 4)
            k_assemble_blocks<4><<<blocks, 256, 0, st>>>(b.nnzb, b.cstart.p, b.contrib.p, b.elems.p, b.emat.p, d_xyz,
                                                         d_lame, n_mat, b.val64.p, flag.p);
        else
            k_assemble_blocks<3><<<blocks, 256, 0, st>>>(b.nnzb, b.cstart.p, b.contrib.p, b.elems.p, b.emat.p, d_xyz,
                                                         d_lame, n_mat, b.val64.p, flag.p);
    }
    const int nblk = (int)std::min<int64_t>((b.n_nodes + 255) / 256, 148 * 16);
    if (b.n_nodes) k_batch_scale<<<nblk, 256, 0, st>>>(b.n_nodes, b.row_ptr.p, b.col.p, b.val64.p, b.dscale.p);
    b.s64_ok = b.s32_ok = false;
    MSFEM_CK(cudaGetLastError());
    return 0;
}

int batch_assemble(BatchSys& b, const double* d_xyz, const double* d_lame, int n_mat)
{
    MSFEM_TRY(batch_assemble_enqueue(b, d_xyz, d_lame, n_mat));
    cudaStream_t st = b.stream;
    int bad = 0;
    MSFEM_CK(cudaMemcpyAsync(&bad, b.aflag.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    MSFEM_CK(cudaStreamSynchronize(st));
    if (bad) {
        set_error("batched systems: material id out of range");
        return MSFEM_ERR_ARGUMENT;
    }
    return 0;
}

int batch_assemble_given(BatchSys& b, const double* d_eblocks, bool scaled)
{
    cudaStream_t st = b.stream;
    MSFEM_TRY(b.val64.alloc(std::max<int64_t>(1, 9 * b.nnzb)));
    if (scaled) {
        MSFEM_TRY(b.dscale.alloc(std::max<int64_t>(1, 3 * b.n_nodes)));
    }
    const int blocks = (int)std::min<int64_t>((b.nnzb + 255) / 256, 148 * 16);
    if (b.nnzb)
        k_assemble_given<<<blocks, 256, 0, st>>>(b.nnzb, b.cstart.p, b.contrib.p, b.k1, d_eblocks, b.val64.p);
    const int nblk = (int)std::min<int64_t>((b.n_nodes + 255) / 256, 148 * 16);
    if (scaled && b.n_nodes)
        k_batch_scale<<<nblk, 256, 0, st>>>(b.n_nodes, b.row_ptr.p, b.col.p, b.val64.p, b.dscale.p);
    b.s64_ok = b.s32_ok = false;
    MSFEM_CK(cudaGetLastError());
    MSFEM_CK(cudaStreamSynchronize(st));
    return 0;
}

}  // namespace msfem
