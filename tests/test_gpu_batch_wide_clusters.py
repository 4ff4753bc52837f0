"""The batched solver (csrc/batch_minres.cu) on wide clusters: several warps per CTA on 8 and 16 CTAs, CTAs
without a single slice (a system much smaller than the batch's largest, whose shares are empty and which so run
ahead of their neighbours), and many refinement steps, each of which sums the residual and then starts the
Krylov sums.  All CTAs of a cluster have to hold the same numbers at each of these: the same bits on every
run, and the oracle's solution.

Tolerance as in tests/test_gpu_batch_cluster.py: 1e-12 on the residual, eigenvalues of the scaled free blocks
above 0.02, 1e-9 on the solution."""
import numpy as np
import pytest

from multiscalefemsolver3d_b200.cells import FP32_IR, FP64
from oracle import cells as oc
from test_gpu_batch_cluster import E, NU, _batch

pytestmark = pytest.mark.gpu


def _cluster(sizes, R, threads, sms=148):
    """launch_shape's rule: the cluster doubles while it has fewer warps than the largest system has slices
    and the batch asks for at most four CTAs per multiprocessor."""
    rows_per_slice = {8: 8, 4: 16, 1: 32}[R]
    slices = max(-(-(n - 1) ** 3 // rows_per_slice) for n in sizes)
    c = 1
    while c < 16 and c * (threads // 32) < slices and len(sizes) * 2 * c <= 4 * sms:
        c *= 2
    return c


# sizes, right-hand sides, threads, the cluster that the rule gives
CASES = [([12], 8, 512, 16), ([14], 4, 512, 16), ([12, 2, 3], 8, 512, 16), ([9, 2, 2, 3], 8, 256, 8),
         ([9, 2, 2, 3], 8, 32, 16), ([8, 2], 1, 64, 8), ([10, 2, 4], 4, 128, 16), ([10, 2, 4], 4, 256, 8)]


@pytest.mark.parametrize("precision", [FP64, FP32_IR], ids=["fp64", "fp32_ir"])
@pytest.mark.parametrize("sizes,R,threads,cluster", CASES, ids=lambda v: str(v).replace(", ", "-").strip("[]"))
def test_wide_clusters(lib, cuda, sizes, R, threads, cluster, precision):
    assert _cluster(sizes, R, threads) == cluster
    b, parts, no, x0 = _batch(3, sizes, R)
    runs = []
    for _ in range(5):
        x, rc = b.solve(x0, precision=precision, tol=1e-12, maxiter=2000, threads=threads)
        rep = b.report()
        assert rc == 0 and rep["rel"].max() <= 1e-12
        runs.append((x, rep["inner"], rep["outer"], rep["rel"]))
    b.close()
    if precision == FP32_IR:
        assert runs[0][2].max() >= 2  # a residual between two inner solves
    for r in runs[1:]:
        for a, first in zip(r, runs[0]):
            np.testing.assert_array_equal(a, first)
    for s in {0, len(sizes) - 1}:
        xyz, el, mat, edge = parts[s]
        fixed = np.nonzero(edge)[0]
        K = oc.assemble(xyz, el, mat, E, NU)
        for r in {0, R - 1}:
            g = x0[no[s]:no[s + 1], r]
            ref = oc.solve_dirichlet(K, xyz.shape[0], fixed, g[fixed])
            np.testing.assert_allclose(runs[0][0][no[s]:no[s + 1], r], ref, rtol=0, atol=1e-9 * np.abs(ref).max())
