"""The grid of the z-marching products (csrc/zmarch_grid.h), whose CTAs each leave one partial sum of MINRES's
inner product: the sizes at which it passes the 2048 entries that the other reductions have, on the CPU from the
header itself, and on the GPU a two-level solve on such a box against the one with the stored matrix."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from multiscalefemsolver3d_b200 import fem, meshgen
from multiscalefemsolver3d_b200.cells import FP64, Cells
from multiscalefemsolver3d_b200.twolevel import TwoLevel

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multiscalefemsolver3d_b200", "csrc")
SHIM = """
#include "zmarch_grid.h"
extern "C" void grid(int nx, int ny, int nz, int ox, int oy, long long slots, int* g)
{
    const msfem::ZmarchGrid z = msfem::zmarch_grid(nx, ny, nz, ox, oy, slots);
    g[0] = z.tiles_x, g[1] = z.tiles_y, g[2] = z.seg_len, g[3] = z.n_seg, g[4] = (int)z.ctas();
}
"""
OX, OY, SLOTS = 15, 7, 296  # the FP64 product: 15 x 7 owned nodes, two CTAs on each of 148 multiprocessors


@pytest.fixture(scope="module")
def grid(tmp_path_factory):
    d = tmp_path_factory.mktemp("zmarch")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(d / "shim.cpp"), "-o",
                    str(d / "shim.so")], check=True)
    f = C.CDLL(str(d / "shim.so")).grid

    def call(nx, ny, nz):
        g = (C.c_int * 5)()
        f(nx, ny, nz, OX, OY, C.c_longlong(SLOTS), g)
        return list(g)
    return call


def _ctas(nx, ny, nz):
    tiles, layers = -(-(nx + 1) // OX) * -(-(ny + 1) // OY), nz + 1
    cost = {}
    for n_seg in range(1, layers + 1):
        length = -(-layers // n_seg)
        segs = -(-layers // length)
        cost.setdefault(-(-tiles * segs // SLOTS) * (length + 1), tiles * segs)
    return cost[min(cost)]


@pytest.mark.parametrize("box", [(n, n, n) for n in (1, 14, 15, 128, *range(160, 261, 20))]
                         + [(512, 512, 8), (272, 248, 8), (1, 300, 5), (300, 1, 1)], ids=lambda b: "x".join(map(str, b)))
def test_grid_covers_the_nodes(grid, box):
    tx, ty, seg_len, n_seg, ctas = grid(*box)
    assert (tx - 1) * OX < box[0] + 1 <= tx * OX and (ty - 1) * OY < box[1] + 1 <= ty * OY
    assert (n_seg - 1) * seg_len < box[2] + 1 <= n_seg * seg_len
    assert ctas == tx * ty * n_seg == _ctas(*box)


def test_grid_has_no_small_bound(grid):
    """No fixed scratch of a few thousand entries holds these: cubes from 161^3, flat boxes earlier."""
    assert grid(160, 160, 160)[4] <= 2048 < grid(161, 161, 161)[4]
    assert grid(168, 168, 168)[4] == 3900 and grid(240, 240, 240)[4] == 6545
    assert grid(512, 512, 8)[4] == 2590 and grid(272, 248, 8)[4] == 2052


def _box_cells(mesh, E, nu, H):
    """Cells of H^3 hexahedra over a Kuhn box (meshgen.cube_cells for cubes)."""
    nx, ny, nz = mesh.meta["box"]
    cx, cy, cz = nx // H, ny // H, nz // H
    a = np.arange(H + 1)
    lk, lj, li = (v.ravel() for v in np.meshgrid(a, a, a, indexing="ij"))
    hk, hj, hi = (v.ravel() for v in np.meshgrid(a[:H], a[:H], a[:H], indexing="ij"))
    local = meshgen.kuhn_box(H, H, H).tets
    xyz, tets, mats, boxes, cng, cvert, color = [], [], [], [], [], [], []
    for c in range(cx * cy * cz):
        ci, cj, ck = c % cx, (c // cx) % cy, c // (cx * cy)
        g = (ci * H + li) + (nx + 1) * ((cj * H + lj) + (ny + 1) * (ck * H + lk))
        hexes = (ci * H + hi) + nx * ((cj * H + hj) + ny * (ck * H + hk))
        te = (hexes[:, None] * 6 + np.arange(6)).ravel()
        x = mesh.xyz[g]
        xyz.append(x)
        tets.append(local)
        mats.append(mesh.mat[te])
        boxes.append(np.stack([x.min(0), x.max(0)], 1).ravel())
        cng.append(g)
        cvert.append([(ci + (v & 1)) + (cx + 1) * ((cj + ((v >> 1) & 1)) + (cy + 1) * (ck + (v >> 2)))
                      for v in range(8)])
        color.append((ci & 1) | ((cj & 1) << 1) | ((ck & 1) << 2))
    n = len(boxes)
    cells = meshgen.CellMeshes(node_off=np.arange(n + 1, dtype=np.int64) * (H + 1) ** 3, xyz=np.concatenate(xyz),
                               tet_off=np.arange(n + 1, dtype=np.int64) * 6 * H ** 3,
                               tets=np.concatenate(tets).astype(np.int32), mat=np.concatenate(mats).astype(np.int32),
                               box=np.array(boxes), E=E, nu=nu, m=np.full(n, H, np.int32))
    return meshgen.CubeCells(cells=cells, cell_node_global=np.concatenate(cng).astype(np.int32),
                             cell_vertex=np.array(cvert, np.int32), cell_color=np.array(color, np.int32),
                             n_coarse_vertices=(cx + 1) * (cy + 1) * (cz + 1))


@pytest.mark.gpu
def test_solve_with_more_ctas_than_2048(cuda, grid):
    """Both solves stop at a relative residual of 1e-10; a plate of 8 layers fixed below is far from
    singular (condition below 1e4 scaled), so the solutions agree to 1e-6 of their norm."""
    box, H = (272, 248, 8), 8
    assert grid(*box)[4] > 2048
    mesh = meshgen.kuhn_box(*box, size=tuple(k / 16.0 for k in box))
    rng = np.random.default_rng(5)
    blocks = rng.integers(0, 2, (2, 62, 68))
    k, j, i = np.meshgrid(*(np.arange(n) // 4 for n in box[::-1]), indexing="ij")
    mesh.mat = np.repeat(blocks[k, j, i].ravel(), 6).astype(np.int32)
    E, nu = np.array([1.0, 10.0]), np.array([0.3, 0.3])
    fixed = meshgen.nodes_on_plane(mesh, 2, 0.0)
    dofs = (3 * fixed[:, None] + np.arange(3)).ravel().astype(np.int32)
    faces, _ = meshgen.boundary_faces_on_plane(mesh, 2, 0.5)
    cc = _box_cells(mesh, E, nu, H)
    at = (7 + 8 * 6) + 272 * (3 + 8 * 1) + 272 * 248 * 5  # hexahedron (7, 3, 5) of cell (6, 1, 0)
    np.testing.assert_array_equal(
        cc.cell_node_global.reshape(-1, (H + 1) ** 3)[40][cc.cells.tets[6 * (7 + 8 * (3 + 8 * 5)):][:6]],
        mesh.tets[6 * at:][:6])
    with fem.System(fem.ELASTIC, mesh.xyz, mesh.tets, mesh.mat) as S, \
            fem.System(fem.ELASTIC, mesh.xyz, mesh.tets, mesh.mat) as K:
        S.set_kuhn_grid(*box)
        K.set_kuhn_grid(*box)
        S.add_traction(faces, np.tile([0.1, 0.0, -1.0], (faces.shape[0], 1)))
        S.assemble_elastic(E, nu)
        K.assemble_elastic_textbook(E, nu)
        for s in (S, K):
            s.apply_dirichlet(dofs, np.zeros(dofs.size), fem.ROW_AND_COLUMN)
        cells = Cells(cc.cells)
        assert cells.build_bases(FP64, tol=1e-8) == 0
        T = TwoLevel(S, cells, cc, dofs)
        T.set_smoother(K, matrix_free=True)
        x = {}
        for on in (False, True):
            T.set_matrix_free(on)
            S.set_x(np.zeros(S.n_rows))
            rel, it, _, rc = T.solve(tol=1e-10, precision=FP64)
            assert rc == 0 and rel <= 1e-10
            x[on] = (it, S.get_x())
        T.close()  # before the systems that it refers to
        cells.close()
        assert np.linalg.norm(x[True][1] - x[False][1]) <= 1e-6 * np.linalg.norm(x[False][1])
        assert abs(x[True][0] - x[False][0]) <= 0.05 * x[False][0] + 2
