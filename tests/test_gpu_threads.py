"""One handle per thread: two threads solve systems of different size with the same method at once, again and
again.  A solver's launch shape (its shared memory above all) is the system's own and no state of the kernel that
the other thread could change.  Every solve gives the bits that it gives alone."""
import threading

import numpy as np
import pytest

from multiscalefemsolver3d_b200 import fem
from test_gpu_cg_forms import _spd

pytestmark = pytest.mark.gpu

SIZES = [(4737, 300), (60000, 400)]


def _system(n, reach):
    A, f = _spd(n, reach, n)
    return fem.System.from_csr(fem.Csr(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, f, np.zeros(n)),
                               F=f, X=np.zeros(n))


@pytest.mark.parametrize("method,precision", [(fem.CG, fem.FP64), (fem.PCG_JACOBI, fem.FP64),
                                              (fem.PCG_JACOBI, fem.FP32_IR), (fem.GMRES, fem.FP64),
                                              (fem.GMRES, fem.FP32_IR)])
def test_solves_on_two_threads(lib, cuda, method, precision):
    systems = [_system(*s) for s in SIZES]

    def solve(S):
        S.set_x(np.zeros(S.n_rows))
        rel, it, rc = S.solve(method, precision, tol=1e-11, maxiter=500, restart=20)
        assert rc == 0
        return S.get_x()

    alone = [solve(S) for S in systems]
    errors = []
    start = threading.Barrier(2)

    def work(k):
        try:
            start.wait(60)
            for _ in range(150):
                np.testing.assert_array_equal(solve(systems[k]), alone[k])
        except Exception as e:  # reported by the main thread
            errors.append(f"system {k}: {e}")

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for S in systems:
        S.close()
    assert not errors, errors
