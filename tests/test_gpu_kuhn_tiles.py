"""The z-marching products (csrc/kuhn25.cuh) at the edges of their tiles of 15 x 7 nodes and of the z
segments: grids one node short of a tile, of one tile and of one more, along x and along y, in FP64 and in
the smoother's scaled FP32 form, against the assembled matrix at the bars of tests/test_gpu_kuhn.py."""
import numpy as np
import pytest

from test_gpu_kuhn import _system, box_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(13, 5, 1), (14, 6, 2), (15, 7, 3), (28, 13, 5), (29, 14, 7), (30, 12, 16), (1, 1, 1),
                               (44, 1, 41), (3, 27, 70)], ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("textbook", [False, True], ids=["reference", "textbook"])
def test_products_at_the_tile_edges(cuda, n, textbook):
    p = box_problem(*n, size=tuple(0.25 * k for k in n) if n[0] % 2 else (1.0, 0.7, 0.4), n_mat=3, seed=sum(n))
    with _system(p, textbook) as S:
        S.set_kuhn_grid(*n)
        rng = np.random.default_rng(7)
        x = rng.normal(size=S.n_rows)
        y, ya = S.kuhn_spmv(x), S.spmv(x)
        assert np.linalg.norm(y - ya) <= 1e-13 * np.linalg.norm(ya)
        assert np.abs(y - ya).max() <= 1e-12 * np.abs(ya).max()
        x32 = x.astype(np.float32)
        y, ya = S.kuhn_spmv_scaled32(x32), S.spmv_scaled32(x32)
        assert np.linalg.norm(y - ya) <= 1e-5 * np.linalg.norm(ya)
        np.testing.assert_array_equal(S.kuhn_spmv_scaled32(x32), y)
