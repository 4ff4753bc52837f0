"""GMRES(m) (csrc/gmres.cu) where a CTA's rows of the work vector, or of it and the basis, come within a few
hundred bytes of the shared memory of a multiprocessor: the kernel's own arrays have to fit beside them.

Sizes: with s bytes for 148 CTAs of ceil(slices / 148) slices, FP32 with restart 71 fills it at 108,929 ...
113,664 rows with the basis, FP64 with restart 13 at 279,425 ... 284,160, restart 50 at 4,219,777 ... 4,224,512
with the work vector alone.  One size within each range and one on either side of the first.

The matrices are diagonally dominant with off-diagonal row sums of at most half the diagonal: a relative
residual of 1e-11 leaves the solution within 1e-10 (x a factor for the largest entry): 1e-9, as in
tests/test_gpu_gmres_shapes.py."""
import numpy as np
import pytest
import scipy.sparse as sp

from multiscalefemsolver3d_b200 import fem

pytestmark = pytest.mark.gpu


def _band(n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = rng.uniform(-1, 1, n - 1), rng.uniform(-1, 1, n - 1)
    d = rng.uniform(0.5, 1.0, n)
    d[1:] += 2.0 * np.abs(lo)
    d[:-1] += 2.0 * np.abs(hi)
    A = sp.diags([lo, d, hi], [-1, 0, 1], format="csr")
    A.sort_indices()
    return A, rng.uniform(-1, 1, n)


@pytest.mark.parametrize("n,m,precision", [(108900, 71, fem.FP32_IR), (110000, 71, fem.FP32_IR), (113700, 71, fem.FP32_IR),
                                           (280000, 13, fem.FP64), (4220000, 50, fem.FP32_IR), (4220000, 50, fem.FP64)])
def test_gmres_at_the_memory_limit(lib, cuda, n, m, precision):
    A, f = _band(n, n + m)
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
