"""The persistent batched solver (csrc/batch_minres.cu) at the edges of its slices and clusters: free
rows 0, 1, one less and one more than a slice, systems of very different sizes in one batch, batches
small and large enough to change the cluster size, every number of right-hand sides, both
precisions and several CTA sizes, against the oracle's exact solution of each system.

Tolerance: the solves stop at a relative residual of 1e-12; the Jacobi-scaled free blocks of these
meshes (E 1:10) have no eigenvalue below 0.02 in modulus, so the solution is within about 5e-11 of the
exact one; 1e-9 leaves a factor for the largest entry against the norm."""
import numpy as np
import pytest

from multiscalefemsolver3d_b200 import meshgen
from multiscalefemsolver3d_b200.cells import FP32_IR, FP64, BatchSystems
from oracle import cells as oc

pytestmark = pytest.mark.gpu

E, NU = np.array([1.0, 10.0]), np.array([0.3, 0.3])


def _cube(n, seed):
    m = meshgen.kuhn_cube(n, jitter=0.1, seed=seed)
    rng = np.random.default_rng(seed)
    inside = ((meshgen.tet_centroids(m) - rng.uniform(0.2, 0.8, 3)) ** 2).sum(1) < 0.12
    edge = ((np.abs(m.xyz) < 1e-12) | (np.abs(m.xyz - 1.0) < 1e-12)).any(1)
    return m.xyz, m.tets.astype(np.int64), inside.astype(np.int32), edge


def _sheet(n, seed):
    """A triangulated unit square in space (z a plane function of x and y)."""
    rng = np.random.default_rng(seed)
    j, i = np.meshgrid(np.arange(n + 1), np.arange(n + 1), indexing="ij")
    x, y = i.ravel() / n, j.ravel() / n
    edge = (i.ravel() % n == 0) | (j.ravel() % n == 0)
    x, y = x + ~edge * rng.uniform(-0.1, 0.1, x.size) / n, y + ~edge * rng.uniform(-0.1, 0.1, x.size) / n
    xyz = np.stack([x, y, 0.3 * x - 0.2 * y], 1)
    a = (np.arange(n)[None, :] + (n + 1) * np.arange(n)[:, None]).ravel()
    tri = np.concatenate([np.stack([a, a + 1, a + n + 2], 1), np.stack([a, a + n + 2, a + n + 1], 1)])
    return xyz, tri.astype(np.int64), rng.integers(0, 2, tri.shape[0]).astype(np.int32), edge


def _batch(dim, sizes, R):
    parts = [(_cube if dim == 3 else _sheet)(n, 10 + k) for k, n in enumerate(sizes)]
    no, eo = [0], [0]
    for xyz, el, _, _ in parts:
        no.append(no[-1] + xyz.shape[0])
        eo.append(eo[-1] + el.shape[0])
    rng = np.random.default_rng(R)
    x = rng.uniform(-1, 1, (no[-1], R, 3))
    fixed = np.concatenate([p[3] for p in parts])
    x[~fixed] = 0.0
    b = BatchSystems(dim, no, np.concatenate([p[0] for p in parts]), eo,
                     np.concatenate([p[1] + o for p, o in zip(parts, no)]), np.concatenate([p[2] for p in parts]), E, NU,
                     fixed, R)
    return b, parts, no, x


def _check(dim, sizes, R, precision, threads, check=None):
    b, parts, no, x0 = _batch(dim, sizes, R)
    x, rc = b.solve(x0, precision=precision, tol=1e-12, maxiter=2000, threads=threads)
    rep = b.report()
    b.close()
    assert rc == 0 and rep["rel"].max() <= 1e-12
    for s in range(len(sizes)) if check is None else check:
        xyz, el, mat, edge = parts[s]
        fixed = np.nonzero(edge)[0]
        K = oc.assemble(xyz, el, mat, E, NU)
        for r in range(R):
            g = x0[no[s]:no[s + 1], r]
            ref = oc.solve_dirichlet(K, xyz.shape[0], fixed, g[fixed])
            np.testing.assert_allclose(x[no[s]:no[s + 1], r], ref, rtol=0, atol=1e-9 * np.abs(ref).max())


# cubes of n hexahedra per edge have (n-1)^3 free rows: 0, 1, 8 (a slice at R = 8), 27, 64, 125, 216
@pytest.mark.parametrize("R", [1, 4, 8])
@pytest.mark.parametrize("precision", [FP64, FP32_IR])
def test_volume_systems_of_every_size(lib, cuda, R, precision):
    _check(3, [5, 1, 2, 7, 3, 4, 6], R, precision, 0)


# sheets have (n-1)^2 free rows: 0, 1, 4, 9, 16 (a slice at R = 4), 25, 36 (past one at R = 1), 169
@pytest.mark.parametrize("R", [1, 4, 8])
def test_face_systems_of_every_size(lib, cuda, R):
    _check(2, [1, 14, 2, 3, 4, 5, 6, 7], R, FP64, 0)


@pytest.mark.parametrize("threads", [32, 96, 512])
def test_cta_sizes(lib, cuda, threads):
    _check(3, [4, 6, 2], 8, FP64, threads)


# 1 and 30 systems run on clusters of several CTAs, 400 on one CTA each
@pytest.mark.parametrize("count", [1, 30, 400])
def test_batches_of_every_cluster_size(lib, cuda, count):
    sizes = [4 + k % 3 for k in range(count)]
    _check(3, sizes, 4, FP64, 64, check=[0, count // 2, count - 1])
