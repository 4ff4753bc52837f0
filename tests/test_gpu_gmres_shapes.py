"""GMRES(m) (csrc/gmres.cu) at the edges of its layout: systems smaller than a slice, one row past a
slice, fewer slices than CTAs, restart depths of 1, past the system's size, and deep enough that
the basis leaves shared memory, 3x3-block rows, both precisions -- against Jacobi iterations to the last
bit (a sparse LU for the block case).

The matrices are diagonally dominant with row sums of off-diagonals at most half the diagonal, so
||A^-1 D|| <= 2 and a relative residual of 1e-11 leaves the solution within 1e-10 (x a factor for the
largest entry): 1e-9."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from multiscalefemsolver3d_b200 import fem, meshgen

pytestmark = pytest.mark.gpu


def _dominant(n, seed, per_row=6):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n), per_row)
    cols = rng.integers(0, n, rows.size)
    A = sp.csr_matrix((rng.uniform(-1, 1, rows.size), (rows, cols)), shape=(n, n))
    A.setdiag(0.0)
    A.eliminate_zeros()
    d = 2.0 * np.asarray(abs(A).sum(axis=1)).ravel() + rng.uniform(0.5, 1.0, n)
    return (A + sp.diags(d)).tocsr(), rng.uniform(-1, 1, n)


@pytest.mark.parametrize("precision", [fem.FP64, fem.FP32_IR])
@pytest.mark.parametrize("n,m", [(1, 1), (2, 5), (31, 1), (33, 50), (4737, 7), (20000, 30), (60000, 300)])
def test_gmres_solution(lib, cuda, n, m, precision):
    A, f = _dominant(n, n + m)
    A.sort_indices()
    S = fem.System.from_csr(fem.Csr(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, f, np.zeros(n)),
                            F=f, X=np.zeros(n))
    rel, it, rc = S.solve(fem.GMRES, precision, tol=1e-11, maxiter=5000, restart=m)
    x = S.get_x()
    S.close()
    d = A.diagonal()
    ref = f / d
    for _ in range(120):  # the error halves at least, every time
        ref = ref + (f - A @ ref) / d
    assert rc == 0 and rel <= 1.0001e-11
    np.testing.assert_allclose(x, ref, rtol=0, atol=1e-9 * np.abs(ref).max())


def test_gmres_block_rows_and_start(lib, cuda):
    """3x3-block rows from a nonzero start, stopped at maxiter and continued to the solution."""
    p = meshgen.cube_elastic(n=6)
    S = fem.System(fem.ELASTIC, p.mesh.xyz, p.mesh.tets, p.mesh.mat)
    S.assemble_elastic_textbook(p.E, p.nu)
    S.add_traction(p.faces, p.traction)
    dofs = (3 * p.bc_nodes[:, None] + np.arange(3)).ravel().astype(np.int32)
    S.apply_dirichlet(dofs, np.zeros(dofs.size), fem.ROW_AND_COLUMN)
    A = S.export_csr()
    rel, it, rc = S.solve(fem.GMRES, fem.FP64, tol=1e-12, maxiter=17, restart=50)
    assert rc == 1 and it == 17
    rel, it, rc = S.solve(fem.GMRES, fem.FP64, tol=1e-12, maxiter=20000, restart=50)
    x = S.get_x()
    S.close()
    assert rc == 0
    ref = spl.spsolve(A.to_scipy().tocsc(), A.F)
    # the scaled matrix's condition is below 1e4 on this cube: 1e-12 residual, 1e-8 solution
    np.testing.assert_allclose(x, ref, rtol=0, atol=1e-8 * np.abs(ref).max())
