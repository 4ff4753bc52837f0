"""GMRES(m) (csrc/gmres.cu) with few vectors and the basis in global memory, where several warps share the rows of a
vector: restart depths 1, 2, 5 (a number that does not divide the 32 warps), 15, 16 and 17 (the first without), the
work vector in shared and in global memory, 3x3-block rows, columns in no order.

The matrices are diagonally dominant with off-diagonal row sums of at most half the diagonal: a relative residual
of 1e-11 leaves the solution within 1e-10 (x a factor for the largest entry): 1e-9, as in
tests/test_gpu_gmres_shapes.py."""
import numpy as np
import pytest

from multiscalefemsolver3d_b200 import fem, meshgen
from test_gpu_gmres_memory import _band
from test_gpu_gmres_shapes import _dominant

pytestmark = pytest.mark.gpu


def _solve(A, f, n, m, precision):
    S = fem.System.from_csr(fem.Csr(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, f, np.zeros(n)),
                            F=f, X=np.zeros(n))
    rel, it, rc = S.solve(fem.GMRES, precision, tol=1e-11, maxiter=5000, restart=m)
    x = S.get_x()
    S.close()
    assert rc == 0 and rel <= 1.0001e-11
    d = A.diagonal()
    ref = f / d
    for _ in range(60):  # the error halves at least, every time
        ref = ref + (f - A @ ref) / d
    np.testing.assert_allclose(x, ref, rtol=0, atol=1e-9 * np.abs(ref).max())


# 1,500,000 rows: the basis leaves shared memory at every depth, the work vector stays; 4,300,000: both leave it
@pytest.mark.parametrize("n,m,precision", [(1500000, m, fem.FP64) for m in (1, 2, 5, 15, 16, 17)]
                         + [(1500000, 16, fem.FP32_IR), (3000000, 2, fem.FP32_IR), (4300000, 5, fem.FP64),
                            (4300000, 16, fem.FP32_IR)])
def test_few_vectors(lib, cuda, n, m, precision):
    _solve(*_band(n, n + m), n, m, precision)


@pytest.mark.parametrize("n,m,precision", [(530000, 5, fem.FP64), (1000000, 5, fem.FP32_IR)])
def test_few_vectors_in_no_order(lib, cuda, n, m, precision):
    A, f = _dominant(n, n, 4)
    A.sort_indices()
    _solve(A, f, n, m, precision)


@pytest.mark.parametrize("precision", [fem.FP64, fem.FP32_IR])
def test_few_vectors_block_rows(lib, cuda, precision):
    """3x3-block rows at 60^3 (680,943 unknowns): the residual that is reported is the solution's."""
    p = meshgen.cube_elastic(n=60)
    S = fem.System(fem.ELASTIC, p.mesh.xyz, p.mesh.tets, p.mesh.mat)
    S.assemble_elastic_textbook(p.E, p.nu)
    S.add_traction(p.faces, p.traction)
    dofs = (3 * p.bc_nodes[:, None] + np.arange(3)).ravel().astype(np.int32)
    S.apply_dirichlet(dofs, np.zeros(dofs.size), fem.ROW_AND_COLUMN)
    x0 = np.zeros(S.n_rows)
    S.set_x(x0)
    r16 = S.solve(fem.GMRES, precision, tol=1e-12, maxiter=160, restart=16)
    x = S.get_x()
    S.set_x(x0)
    r5 = S.solve(fem.GMRES, precision, tol=1e-12, maxiter=160, restart=5)
    A = S.export_csr()
    S.close()
    assert r16[1] == r5[1] == 160 and r16[0] < r5[0] < 1.0  # the deeper restart is further after as many steps
    r = A.F - A.to_scipy() @ x
    assert abs(np.linalg.norm(r) / np.linalg.norm(A.F) / r16[0] - 1.0) <= 1e-6
