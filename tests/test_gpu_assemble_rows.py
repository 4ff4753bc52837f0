"""The row-gathering assembly (csrc/assemble.cu) where its loops take a second turn: a fan of
tetrahedra around one node, whose row has more than 32 entries and whose element list is longer than a
warp, up to the largest degree the portrait accepts (64) -- every kind of element, against the
restated element matrices summed by scipy.  Both sum at most 64 terms per entry: 64 * 2^-53 of the
largest term, below 1e-13 of the largest entry; 1e-12 as in the other parity tests."""
import numpy as np
import pytest
import scipy.sparse as sp
from scipy.spatial import ConvexHull

from multiscalefemsolver3d_b200 import fem
from multiscalefemsolver3d_b200._lib import MsfemError
from oracle import cells as oc

pytestmark = pytest.mark.gpu


def _fan(points):
    """`points` sphere nodes and a centre: 2 * points - 4 tetrahedra share the centre, which is the
    last node, so its row is the longest."""
    k = np.arange(points) + 0.5
    phi, th = np.arccos(1 - 2 * k / points), np.pi * (1 + 5 ** 0.5) * k
    xyz = np.stack([np.cos(th) * np.sin(phi), np.sin(th) * np.sin(phi), np.cos(phi)], 1)
    tri = ConvexHull(xyz).simplices
    tets = np.concatenate([np.full((tri.shape[0], 1), points), tri], 1)
    rng = np.random.default_rng(points)
    for t in tets:
        rng.shuffle(t)
    rng.shuffle(tets)
    return np.concatenate([xyz, [[0.1, -0.05, 0.07]]]), tets.astype(np.int32), rng.integers(0, 2, tets.shape[0]).astype(np.int32)


def _scalar(xyz, tets, S, M):
    g = np.empty((tets.shape[0], 4, 3))
    V = np.empty(tets.shape[0])
    for e, t in enumerate(tets):
        g[e], V[e] = oc.simplex_gradients(xyz[t])
    K = V[:, None, None] * (S[:, None, None] * np.einsum("eia,eja->eij", g, g) + M[:, None, None] / 16)
    n = xyz.shape[0]
    r, c = np.repeat(tets, 4, axis=1).ravel(), np.tile(tets, (1, 4)).ravel()
    return sp.csr_matrix((K.ravel(), (r, c)), shape=(n, n)), V


def _close(A, B):
    D = A.to_scipy()
    assert abs(D - B).max() <= 1e-12 * abs(B).max()


# 18 points: 32 elements, a full warp; 19: one more; 34: 64 elements, the largest degree; rows 19 .. 35
@pytest.mark.parametrize("points", [18, 19, 32, 34])
def test_rows_longer_than_a_warp(lib, cuda, points):
    xyz, tets, mat = _fan(points)
    E, nu = np.array([1.0, 7.0]), np.array([0.3, 0.2])
    for textbook in (False, True):
        S = fem.System(fem.ELASTIC, xyz, tets, mat)
        (S.assemble_elastic_textbook if textbook else S.assemble_elastic)(E, nu)
        _close(S.export_csr(), oc.assemble(xyz, tets, mat, E, nu, textbook=textbook))
        S.assemble_elastic(E, nu)  # a second assembly adds to the first
        _close(S.export_csr(), oc.assemble(xyz, tets, mat, E, nu, textbook=textbook) + oc.assemble(xyz, tets, mat, E, nu))
        S.close()
    sig = np.array([2.0, 5.0])
    S = fem.System(fem.SCALAR, xyz, tets, mat)
    S.assemble_scalar(sig)
    B, _ = _scalar(xyz, tets, sig[mat], np.zeros(mat.size))
    _close(S.export_csr(), B)
    S.close()
    rng = np.random.default_rng(1)
    s, m, f = (rng.uniform(0.5, 2.0, mat.size) for _ in range(3))
    S = fem.System(fem.SCALAR, xyz, tets, mat)
    S.assemble_scalar3(s, m, f)
    B, V = _scalar(xyz, tets, s, m)
    A = S.export_csr()
    _close(A, B)
    F = np.zeros(xyz.shape[0])
    np.add.at(F, tets.ravel(), np.repeat(f * V / 4, 4))
    np.testing.assert_allclose(A.F, F, rtol=0, atol=1e-12 * np.abs(F).max())
    S.close()


def test_degree_limit(lib, cuda):
    xyz, tets, mat = _fan(35)
    with pytest.raises(MsfemError):
        fem.System(fem.SCALAR, xyz, tets, mat)
