// Batches of independent 3x3-block elasticity systems: the MsFEM cell
// sub-problems (faces and volumes of every macro cell) solved together.
#pragma once

#include <vector>

#include "internal.cuh"

namespace msfem {

// n_sys systems on one node numbering: system s owns nodes [node_off[s],
// node_off[s+1]) and elements [elem_off[s], elem_off[s+1]) whose node ids lie in
// its own range.  Matrix: node-level CSR of 3x3 blocks (global column ids), rows
// sorted, diagonal included, built by one stable sort of every element's
// (row, column) pairs; `contrib` keeps the sorted pairs so that each block is
// the sum of its element contributions in element order.
struct BatchSys {
    int dim = 3;  // 2: triangles, 3: tetrahedra
    int k1 = 4;   // nodes per element (at most 32)
    int n_sys = 0;
    int R = 1;    // right-hand sides per system
    int64_t n_nodes = 0, n_elems = 0, nnzb = 0, n_pairs = 0;
    int max_nodes = 0;
    cudaStream_t stream = nullptr;  // the owner's stream
    std::vector<int64_t> h_node_off, h_elem_off;

    DBuf<int64_t> node_off, elem_off;
    DBuf<int32_t> elems;     // [n_elems * k1] global node ids
    DBuf<int32_t> emat;      // [n_elems]
    DBuf<uint8_t> fixed;     // [n_nodes] 1 = Dirichlet node (all three components)
    DBuf<int64_t> row_ptr;   // [n_nodes + 1]
    DBuf<int64_t> cstart;    // [nnzb + 1] first contribution of each block
    DBuf<int32_t> col;       // [nnzb]
    DBuf<uint32_t> contrib;  // [n_pairs] element << 4 | I << 2 | J, grouped by block, element order
    DBuf<double> val64;      // [9 * nnzb] A[a][b] of each block, row-major
    DBuf<double> dscale;     // [3 * n_nodes] 1 / sqrt(diagonal)
    DBuf<int32_t> order;     // systems, largest first (the persistent solver's queue)

    // the free block S A_II S in slices of G rows (batch_minres.cu): rows and columns are the system's
    // free nodes; entry (slice s, position k, row g) has its column at (slice_ptr[s] + k) * G + g and
    // its 9 values at ((slice_ptr[s] + k) * 9 + e) * G + g; shorter rows end in zero blocks
    int64_t n_slices = 0, n_entries = 0;
    int max_slices = 0;        // slices of the largest system
    DBuf<int64_t> slice_off;   // [n_sys + 1]
    DBuf<int64_t> slice_ptr;   // [n_slices + 1]
    DBuf<int32_t> free_node;   // [n_slices * G] node of each free row, -1 past a system's last
    DBuf<int32_t> lid;         // [n_nodes] free row of a node within its system, -1: Dirichlet
    DBuf<int32_t> scol;
    DBuf<double> s64;
    DBuf<float> s32;
    bool s64_ok = false, s32_ok = false;  // they hold the current values

    // solver scratch and per-system report
    DBuf<unsigned char> work;  // Krylov vectors of each cluster (bytes: room for FP64)
    DBuf<int> queue;
    DBuf<int32_t> iters, outers;
    DBuf<double> rel;
    const double* rhs = nullptr;  // optional source term [n_nodes][R][3] (device), used by batch_solve
    int threads = 0;  // CTA size of the last solve
    float last_ms = 0.f;
    DBuf<int> aflag;  // set by the assembly when an element's material id is out of range
};

// pattern: elems/emat/node_off/elem_off/fixed filled; builds row_ptr, col, cstart, contrib
int batch_build_pattern(BatchSys& b, const double* d_xyz);
// values from the current materials (lame: [n_mat][2] lambda, mu on the device)
int batch_assemble(BatchSys& b, const double* d_xyz, const double* d_lame, int n_mat);
// the same launches without waiting for them (no host synchronisation, no allocation once the
// buffers exist): capturable into a CUDA graph; a bad material id is left in b.aflag
int batch_assemble_enqueue(BatchSys& b, const double* d_xyz, const double* d_lame, int n_mat);
// values from caller-given element blocks [n_elems][k1][k1][9] (device), each block the sum of
// its element contributions in element order; scaled: also the Jacobi scale the
// batched solver reads
int batch_assemble_given(BatchSys& b, const double* d_eblocks, bool scaled = true);
// the free block's pattern (batch_build_pattern calls it when the fixed nodes are known)
int batch_build_free(BatchSys& b);
// solves every system; x: [n_nodes][R][3] FP64, fixed entries hold the Dirichlet data on
// entry, free entries are overwritten.  precision: MSFEM_FP64 or MSFEM_FP32_IR.  threads <= 0:
// the CTA size is chosen from the batch's sizes.  No host synchronisation, and no allocation from
// the second call with the same precision on: capturable into a CUDA graph.
int batch_solve(BatchSys& b, double* d_x, int precision, double tol, int maxiter, int threads);
// the CTA size batch_solve uses with `threads`
int batch_threads(const BatchSys& b, int threads);

}  // namespace msfem
