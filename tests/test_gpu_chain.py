"""The two-level cycle as a chain of kernels that start before their predecessor has ended
(launch_chained, csrc/devutil.cuh): each must still read what the one before it wrote.  A missing
wait shows as a wrong or an unrepeatable result, so both are checked, on short and long chains
(a smoother of one step leaves no product between the entry and the residual), with the products
formed from the grid and from the stored matrices."""
import numpy as np
import pytest
import scipy.sparse.linalg as spl

from multiscalefemsolver3d_b200 import fem
from multiscalefemsolver3d_b200.cells import FP64
from multiscalefemsolver3d_b200.twolevel import TwoLevel
from test_gpu_twolevel import _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [1, 2, 4])
@pytest.mark.parametrize("matrix_free", [True, False], ids=["matrix-free", "stored"])
def test_chained_cycle(cuda, degree, matrix_free):
    """The inner tolerance 1e-12 is on the residual; the solution is held to 1e-8 as for the cycle's
    other solves, and a second solve gives the same bits in the same number of iterations."""
    p, S, cc, cells, dofs = _setup()
    with fem.System(fem.ELASTIC, p.mesh.xyz, p.mesh.tets, p.mesh.mat) as K:
        K.assemble_elastic_textbook(p.E, p.nu)
        K.apply_dirichlet(dofs, np.zeros(dofs.size), fem.ROW_AND_COLUMN)
        T = TwoLevel(S, cells, cc, dofs)
        if matrix_free:
            S.set_kuhn_grid(p.mesh.n)
            K.set_kuhn_grid(p.mesh.n)
        T.set_smoother(K, degree=degree, ratio=30.0, matrix_free=matrix_free)
        T.set_matrix_free(matrix_free)
        A = S.export_csr()
        x_exact = spl.spsolve(A.to_scipy().tocsc(), A.F)
        runs = []
        for _ in range(2):
            S.set_x(np.zeros(A.n))
            rel, it, _, rc = T.solve(tol=1e-12, maxiter=20000, precision=FP64)
            assert rc == 0 and rel <= 1e-12
            runs.append((it, S.get_x()))
        assert np.linalg.norm(runs[0][1] - x_exact) <= 1e-8 * np.linalg.norm(x_exact)
        assert runs[0][0] == runs[1][0]
        np.testing.assert_array_equal(runs[0][1], runs[1][1])
