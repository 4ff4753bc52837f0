"""total_launches of a two-level solve: every kernel of the iterations that it replays.  A solve held to one
iteration replays 64 (four graphs of 16) and launches a few kernels beside them, fewer than 64: the whole part of
the difference by 64 is the kernels of an iteration.  A step that raised the residual is taken again with a wider
spectrum bound, which the statistics count."""
import numpy as np
import pytest

from multiscalefemsolver3d_b200 import fem
from multiscalefemsolver3d_b200.cells import FP32_IR, FP64
from multiscalefemsolver3d_b200.twolevel import TwoLevel
from test_gpu_twolevel import _setup

pytestmark = pytest.mark.gpu


def _per_iteration(S, T, precision):
    S.set_x(np.zeros(S.n_rows))
    before, widened = S.stats()["total_launches"], T.stats()["widened"]
    T.solve(tol=1e-12, maxiter=1, precision=precision)
    solves = 1 + T.stats()["widened"] - widened
    return (S.stats()["total_launches"] - before) // (64 * solves)


def test_launches_of_an_iteration(lib, cuda):
    p, S, cc, cells, dofs = _setup()
    with fem.System(fem.ELASTIC, p.mesh.xyz, p.mesh.tets, p.mesh.mat) as K:
        K.assemble_elastic_textbook(p.E, p.nu)
        K.apply_dirichlet(dofs, np.zeros(dofs.size), fem.ROW_AND_COLUMN)
        T = TwoLevel(S, cells, cc, dofs)
        # product, restriction, gather, coarse product and its sums, prolongation, update
        assert _per_iteration(S, T, FP32_IR) == 7
        assert _per_iteration(S, T, FP64) == 7
        S.set_kuhn_grid(p.mesh.n)
        K.set_kuhn_grid(p.mesh.n)
        for matrix_free in (False, True):
            for degree in (1, 4, 5):
                T.set_smoother(K, degree=degree, ratio=30.0, matrix_free=matrix_free)
                T.set_matrix_free(matrix_free)
                # product, entry, two residuals, restriction, gather, coarse product and its sums, prolongation, exit,
                # update, and the steps of the two smoothings after their first
                assert _per_iteration(S, T, FP64) == 11 + 2 * (degree - 1)
        T.close()
