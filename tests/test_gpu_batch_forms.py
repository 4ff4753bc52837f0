"""The batched solver (csrc/batch_minres.cu) with one CTA a system: systems of 0, 1, 2, 8 and 9 slices, on either
side of the form whose matrix stays in the L1, fewer slices than warps and more, batches too large for clusters,
every number of right-hand sides, both precisions; and the same bits whatever the batch around a system is.

Tolerance as in tests/test_gpu_batch_cluster.py: 1e-12 on the residual, eigenvalues of the scaled free blocks above
0.02, 1e-9 on the solution."""
import numpy as np
import pytest

from multiscalefemsolver3d_b200.cells import FP32_IR, FP64
from test_gpu_batch_cluster import _batch, _check

pytestmark = pytest.mark.gpu


# sheets of n squares per edge have (n - 1)^2 free rows; slices of 32, 16, 8 rows at R = 1, 4, 8: within 8 slices and 128
# rows with the first two batches of each (100 rows in 4 slices, 121 in 8, 64 in 8), past it with the others
@pytest.mark.parametrize("R,sizes", [(1, [1, 2, 3]), (1, [11, 2, 6]), (1, [17, 2, 6]), (1, [18, 1, 7]), (4, [1, 2, 5]), (4, [12, 5, 6]),
                                     (4, [13, 3, 9]), (8, [2, 1, 3]), (8, [9, 2, 4]), (8, [10, 5, 2])])
@pytest.mark.parametrize("precision", [FP64, FP32_IR], ids=["fp64", "fp32_ir"])
def test_small_sheets(lib, cuda, R, sizes, precision):
    _check(2, sizes, R, precision, 0)


# 300 systems ask for two CTAs an SM: one CTA each, whatever their size
@pytest.mark.parametrize("R", [1, 4, 8])
@pytest.mark.parametrize("precision", [FP64, FP32_IR], ids=["fp64", "fp32_ir"])
def test_many_cubes(lib, cuda, R, precision):
    _check(3, [(3, 7, 2, 5)[k % 4] for k in range(300)], R, precision, 0, check=[0, 1, 151, 299])


@pytest.mark.parametrize("precision", [FP64, FP32_IR], ids=["fp64", "fp32_ir"])
def test_bits_do_not_depend_on_the_batch(lib, cuda, precision):
    """A batch of 4 small sheets and one of 600 with the same 4 in front: same form, same bits."""
    sizes = [5, 2, 8, 3]
    out = []
    for count in (4, 600):
        b, parts, no, x0 = _batch(2, [sizes[k % 4] for k in range(count)], 4)
        x0 = x0.copy()
        if out:
            x0[:no[4]] = first
        else:
            first = x0[:no[4]].copy()
        x, rc = b.solve(x0, precision=precision, tol=1e-12, maxiter=2000)
        assert rc == 0
        b.close()
        out.append(x[:no[4]])
    np.testing.assert_array_equal(out[0], out[1])
