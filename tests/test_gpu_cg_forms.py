"""CG in one cooperative launch (csrc/krylov_coop.cu) at the edges of its forms: systems smaller than a
slice, one row past a slice, one slice per CTA and one more, a matrix share that fits shared memory
and one that does not, columns too far apart for a window and for 16-bit deltas, 3x3 blocks -- plain CG,
Jacobi-PCG in FP64 and FP32 refinement, against Jacobi iterations to the last bit.

The matrices are symmetric and diagonally dominant with off-diagonal row sums of at most half the
diagonal: ||A^-1 D|| <= 2, so a relative residual of 1e-12 leaves the solution within 1e-11 (times a
factor for the largest entry): 1e-9."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from multiscalefemsolver3d_b200 import fem, meshgen

pytestmark = pytest.mark.gpu


def _spd(n, reach, seed, per_row=4):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n), per_row)
    cols = np.clip(rows + rng.integers(-reach, reach + 1, rows.size), 0, n - 1)
    A = sp.csr_matrix((rng.uniform(-1, 1, rows.size), (rows, cols)), shape=(n, n))
    A = (A + A.T).tocsr()
    A.setdiag(0.0)
    A.eliminate_zeros()
    d = 2.0 * np.asarray(abs(A).sum(axis=1)).ravel() + rng.uniform(0.5, 1.0, n)
    A = (A + sp.diags(d)).tocsr()
    A.sort_indices()
    return A, rng.uniform(-1, 1, n)


# 4736 rows: one slice on each of 148 SMs, 4737: one more; 60,000: several slices, still resident;
# 400,000: streamed; reach 40,000: beyond 16-bit deltas, and a window past shared memory at the last size
@pytest.mark.parametrize("method,precision", [(fem.CG, fem.FP64), (fem.PCG_JACOBI, fem.FP64), (fem.PCG_JACOBI, fem.FP32_IR)])
@pytest.mark.parametrize("n,reach", [(1, 1), (2, 1), (31, 5), (33, 40), (4736, 50), (4737, 4737), (60000, 400),
                                     (60000, 40000), (400000, 3000), (400000, 40000)])
def test_cg_solution(lib, cuda, n, reach, method, precision):
    A, f = _spd(n, reach, n + reach)
    S = fem.System.from_csr(fem.Csr(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, f, np.zeros(n)),
                            F=f, X=np.zeros(n))
    rel, it, rc = S.solve(method, precision, tol=1e-12, maxiter=5000)
    x = S.get_x()
    S.close()
    d = A.diagonal()
    ref = f / d
    for _ in range(120):  # the error halves at least, every time
        ref = ref + (f - A @ ref) / d
    assert rc == 0 and rel <= 1.5e-12
    np.testing.assert_allclose(x, ref, rtol=0, atol=1e-9 * np.abs(ref).max())


@pytest.mark.parametrize("n", [3, 17, 30])
@pytest.mark.parametrize("precision", [fem.FP64, fem.FP32_IR])
def test_cg_block_rows(lib, cuda, n, precision):
    """3x3-block rows: 2, 183 and 931 slices (one per CTA, resident shares, and in FP64 at 30 a streamed
    one), stopped at maxiter and continued."""
    p = meshgen.cube_elastic(n=n)
    S = fem.System(fem.ELASTIC, p.mesh.xyz, p.mesh.tets, p.mesh.mat)
    S.assemble_elastic_textbook(p.E, p.nu)
    S.add_traction(p.faces, p.traction)
    dofs = (3 * p.bc_nodes[:, None] + np.arange(3)).ravel().astype(np.int32)
    S.apply_dirichlet(dofs, np.zeros(dofs.size), fem.ROW_AND_COLUMN)
    rel, it, rc = S.solve(fem.PCG_JACOBI, fem.FP64, tol=1e-12, maxiter=7)
    assert rc == 1 and it == 7
    rel, it, rc = S.solve(fem.PCG_JACOBI, precision, tol=1e-11, maxiter=20000)
    x, A = S.get_x(), S.export_csr()
    S.close()
    assert rc == 0
    if n <= 17:
        ref = spl.spsolve(A.to_scipy().tocsc(), A.F)
        # condition of the scaled matrix below 1e4: 1e-11 residual, 1e-7 solution at worst
        np.testing.assert_allclose(x, ref, rtol=0, atol=1e-7 * np.abs(ref).max())
    r = A.F - A.to_scipy() @ x
    assert np.linalg.norm(r) <= 2e-11 * np.linalg.norm(A.F)
