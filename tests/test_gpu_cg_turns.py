"""CG in one cooperative launch (csrc/krylov_coop.cu) on scalar systems whose CTAs, each with a range of rows of its
own, would gather through windows that together exceed the L2 -- the grid then takes the rows in turn -- and on
columns in no order, where fewer vectors lie in shared memory.  Sizes at the edges of a turn of 148 x 1024 rows, of
a slice and of the rule.

Matrices, oracle and tolerance as in tests/test_gpu_cg_forms.py: ||A^-1 D|| <= 2, a relative residual of 1e-12 leaves
the solution within 1e-11 (times a factor for the largest entry): 1e-9."""
import numpy as np
import pytest
import scipy.sparse as sp

from multiscalefemsolver3d_b200 import fem
from test_gpu_cg_forms import _spd

pytestmark = pytest.mark.gpu

TURN = 148 * 1024


# a window is about 2 reach + the range's rows: 148 of them exceed 126 MB from 112,000 (FP64) and 223,000 (FP32) rows on
@pytest.mark.parametrize("n,reach,method,precision", [
    (2 * TURN - 1, 60000, fem.CG, fem.FP64), (2 * TURN + 1, 60000, fem.PCG_JACOBI, fem.FP64),
    (3 * TURN + 33, 60000, fem.PCG_JACOBI, fem.FP64), (300001, 50000, fem.CG, fem.FP64),
    (4 * TURN, 125000, fem.PCG_JACOBI, fem.FP32_IR), (4 * TURN + 1, 125000, fem.PCG_JACOBI, fem.FP32_IR),
    (400001, 400000, fem.CG, fem.FP64), (400001, 400000, fem.PCG_JACOBI, fem.FP32_IR)])
def test_rows_in_turn_and_scattered(lib, cuda, n, reach, method, precision):
    A, f = _spd(n, reach, n + reach)
    S = fem.System.from_csr(fem.Csr(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, f, np.zeros(n)),
                            F=f, X=np.zeros(n))
    rel, it, rc = S.solve(method, precision, tol=1e-12, maxiter=5000)
    x = S.get_x()
    rel2, it2, rc2 = S.solve(method, precision, tol=1e-12, maxiter=5000)  # from the solution
    S.close()
    d = A.diagonal()
    ref = f / d
    for _ in range(120):  # the error halves at least, every time
        ref = ref + (f - A @ ref) / d
    # CG stops by its recursive residual; without a preconditioner, over 110 iterations on this scaling, the true one
    # has drifted from it by up to its own size, as it does with a launch per kernel (1.8e-12 at reach 300,000)
    assert rc == 0 and rc2 == 0 and it2 <= it
    assert method == fem.CG or rel <= 1.5e-12
    np.testing.assert_allclose(x, ref, rtol=0, atol=1e-9 * np.abs(ref).max())


@pytest.mark.parametrize("method,precision", [(fem.CG, fem.FP64), (fem.PCG_JACOBI, fem.FP32_IR), (fem.GMRES, fem.FP64)])
@pytest.mark.parametrize("share", [0.01, 0.9])
def test_local_columns_and_far_ones(lib, cuda, share, method, precision):
    """A spatial order with a share of the rows coupled to the last ones, as enriched unknowns are: a few such rows
    leave the order what it is, most rows make it none."""
    n, reach = 150000, 300
    A, f = _spd(n, reach, 5)
    rng = np.random.default_rng(6)
    far = rng.choice(n // 2, int(share * n // 2), replace=False)
    B = sp.csr_matrix((rng.uniform(-1, 1, far.size), (far, n - 1 - rng.integers(0, n // 100, far.size))), shape=(n, n))
    A = A + B + B.T
    d = 2.0 * (np.asarray(abs(A).sum(axis=1)).ravel() - A.diagonal()) + 0.7
    A.setdiag(d)
    A = A.tocsr()
    A.sort_indices()
    S = fem.System.from_csr(fem.Csr(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, f, np.zeros(n)),
                            F=f, X=np.zeros(n))
    rel, it, rc = S.solve(method, precision, tol=1e-12, maxiter=5000, restart=50)
    x = S.get_x()
    S.close()
    assert rc == 0
    ref = f / d
    for _ in range(120):
        ref = ref + (f - A @ ref) / d
    np.testing.assert_allclose(x, ref, rtol=0, atol=1e-9 * np.abs(ref).max())
