"""What the framework's users run, as measurable cases: for each, the inputs a program has in hand
(`prepare`), one pass through the public entry points (`run`), the bytes and operations the pass
cannot do without (`work`), and the same result from plain torch in 64 bits (`exact`).

The kinds of case:

  potential         an assembled electrostatics / conduction system whose coefficients change: values
                    cleared, assembled, Dirichlet rows and columns, CG solve, solution read
  potential_driver  the one-call scalar driver on host arrays (mesh in, solution out)
  elastic_driver    the one-call elasticity driver on host arrays
  product           y = A x with an assembled elasticity matrix
  bases             MsFEM Order1 cell bases: every edge, face and volume problem of a set of cells
  twolevel          the fine elasticity solve with the MsFEM two-level preconditioner, matrix-free
  cracked           cracked conduction: enriched assembly from host arrays, GMRES(50) solve
  predict           the learned coarse space: bases of a set of cells from the network
  gradient          one forward and backward pass of the network on a training batch

Solves run to 1e-11 ... 1e-13 (the reference's cell drivers ask for 5e-15) on moduli of 1:10, so that a
solution is determined to well below 1e-9 by its inputs: the reference's elasticity matrices turn
indefinite at higher contrasts, and single cells then come close to singular.
"""
from __future__ import annotations

import ctypes as C
import math
from functools import lru_cache

import numpy as np
import torch

from multiscalefemsolver3d_b200 import fem, meshgen, xfem
from multiscalefemsolver3d_b200._lib import check, load
from multiscalefemsolver3d_b200.cells import Cells
from multiscalefemsolver3d_b200.learned import CoarseNet
from multiscalefemsolver3d_b200.twolevel import TwoLevel

DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------------------ the cases

def listed():
    return [
        # a small conduction problem in a parameter loop: launches and latency count
        {"name": "potential_20", "kind": "potential", "n": 20, "jitter": 0.1, "spheres": 8, "precision": "fp64"},
        # the electrostatics workload at its own size: 100^3, permittivity 1:100
        {"name": "potential_100", "kind": "potential", "n": 100, "jitter": 0.0, "spheres": 200, "precision": "fp32_ir"},
        # the electrostatics driver called from a program that holds host arrays
        {"name": "potential_driver_60", "kind": "potential_driver", "n": 60, "spheres": 100, "precision": "fp32_ir"},
        # the elasticity driver on the 20^3 jittered cube, the reference's own kind of run
        {"name": "elastic_driver_20", "kind": "elastic_driver", "n": 20, "jitter": 0.1},
        # residuals and checks with an assembled elasticity matrix
        {"name": "product_63", "kind": "product", "n": 63},
        # one cell re-solved exactly (the learned coarse space's fallback)
        {"name": "bases_1", "kind": "bases", "cells": 1, "edges": "8"},
        # a few macro cells of mixed resolution
        {"name": "bases_8", "kind": "bases", "cells": 8, "edges": "8,12,16,20"},
        # a macro mesh of 4^3 cells of mixed resolution, odd ones among them
        {"name": "bases_64", "kind": "bases", "cells": 64, "edges": "8,11,12,16,17"},
        # the flagship solve: heterogeneous elasticity with the multiplicative two-level cycle
        {"name": "twolevel_40", "kind": "twolevel", "n": 40},
        # cracked conduction, from mesh and cracks to the solution
        {"name": "cracked_40", "kind": "cracked", "n": 40, "cracks": 30},
        # the coarse space of an 8 x 8 x 8 macro mesh predicted by the network
        {"name": "predict_512", "kind": "predict", "cells": 512},
        # a training batch of the network, forward and backward
        {"name": "gradient_128", "kind": "gradient", "cells": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["potential", "potential_driver", "elastic_driver", "product", "bases", "twolevel", "cracked",
                       "predict", "gradient"])
    if kind == "potential":
        n = _log_int(rng, 14, 100)
        return {"kind": kind, "n": n, "jitter": rng.choice([0.0, 0.05, 0.1]), "spheres": rng.randint(4, 200),
                "precision": rng.choice(["fp64", "fp32_ir"])}
    if kind == "potential_driver":
        return {"kind": kind, "n": _log_int(rng, 16, 60), "spheres": rng.randint(4, 100),
                "precision": rng.choice(["fp64", "fp32_ir"])}
    if kind == "elastic_driver":
        return {"kind": kind, "n": rng.randint(10, 20), "jitter": round(rng.uniform(0.02, 0.12), 3)}
    if kind == "product":
        return {"kind": kind, "n": _log_int(rng, 17, 63)}
    if kind == "bases":
        k = rng.randint(1, 4)
        return {"kind": kind, "cells": _log_int(rng, 1, 48),
                "edges": ",".join(str(rng.randint(7, 17)) for _ in range(k))}
    if kind == "twolevel":
        return {"kind": kind, "n": 8 * rng.randint(3, 5)}
    if kind == "cracked":
        return {"kind": kind, "n": rng.randint(20, 40), "cracks": rng.randint(5, 30)}
    if kind == "predict":
        return {"kind": kind, "cells": _log_int(rng, 9, 512)}
    return {"kind": kind, "cells": _log_int(rng, 9, 128)}


# ------------------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _grid_tets(n):
    """int32 [6 n^3, 4] on the GPU: n^3 hexahedra of six Kuhn tetrahedra, x fastest."""
    c = torch.arange(n, device=DEV)
    k, j, i = torch.meshgrid(c, c, c, indexing="ij")
    base = (i + (n + 1) * (j + (n + 1) * k)).reshape(-1, 1)
    off = torch.tensor([(b & 1) + (n + 1) * (((b >> 1) & 1) + (n + 1) * (b >> 2)) for b in range(8)], device=DEV)
    kuhn = torch.tensor([[0, 1, 3, 7], [0, 1, 5, 7], [0, 2, 3, 7], [0, 2, 6, 7], [0, 4, 5, 7], [0, 4, 6, 7]], device=DEV)
    return (base + off)[:, kuhn].reshape(-1, 4).to(torch.int32)


def _cube(n, jitter, seed):
    """(xyz f64 [(n+1)^3, 3], tets) of the unit cube; interior nodes jittered by +-jitter h."""
    g = torch.arange(n + 1, device=DEV, dtype=F64) / n
    k, j, i = torch.meshgrid(g, g, g, indexing="ij")
    xyz = torch.stack([i.reshape(-1), j.reshape(-1), k.reshape(-1)], 1)
    if jitter:
        inner = ((xyz > 1e-9) & (xyz < 1 - 1e-9)).all(1, keepdim=True)
        off = (torch.rand(xyz.shape, generator=_gen(seed), device=DEV, dtype=F64) * 2 - 1) * (jitter / n)
        xyz = xyz + torch.where(inner, off, torch.zeros_like(off))
    return xyz.contiguous(), _grid_tets(n)


def _marked(xyz, tets, count, rmin, rmax, seed):
    """int32 material per tetrahedron: 1 where its centroid lies in one of `count` random spheres."""
    rng = np.random.default_rng(seed)
    c = torch.from_numpy(rng.uniform(0.0, 1.0, (count, 3))).to(DEV)
    r2 = torch.from_numpy(rng.uniform(rmin, rmax, count) ** 2).to(DEV)
    cen = xyz[tets.long()].mean(1)
    inside = torch.zeros(tets.shape[0], dtype=torch.bool, device=DEV)
    for k in range(count):
        inside |= ((cen - c[k]) ** 2).sum(1) < r2[k]
    return inside.to(torch.int32)


def _potential_inputs(case, seed):
    n = case["n"]
    xyz, tets = _cube(n, case.get("jitter", 0.0), seed)
    mat = _marked(xyz, tets, case["spheres"], 0.02, 0.06 if n > 40 else 0.15, seed)
    node = torch.arange((n + 1) ** 3, device=DEV)
    left, right = node[node % (n + 1) == 0], node[node % (n + 1) == n]
    nodes = torch.cat([left, right]).to(torch.int32)
    values = torch.cat([torch.ones(left.numel()), torch.zeros(right.numel())]).to(DEV, F64)
    sigma = np.array([1.0, np.random.default_rng(seed).uniform(50.0, 150.0)])
    return xyz, tets, mat, sigma, nodes, values


def _elastic_inputs(n, jitter, seed):
    """Cube with u = 0 on z = 0 and a traction on z = 1: (xyz, tets, fixed nodes, top faces, traction)."""
    xyz, tets = _cube(n, jitter, seed)
    plane = (n + 1) ** 2
    fixed = torch.arange(plane, device=DEV, dtype=torch.int32)
    t = tets.long()
    on = t >= plane * n
    hit = on.sum(1) == 3
    faces = t[hit][on[hit]].reshape(-1, 3).to(torch.int32)
    rng = np.random.default_rng(seed)
    load_ = np.tile(np.array([0.0, 0.0, -1.0]) + rng.uniform(-0.2, 0.2, 3), (faces.shape[0], 1))
    return xyz, tets, fixed, faces, load_


def _host(t):
    return t.cpu().numpy()


@lru_cache(maxsize=32)
def _cell_template(m):
    t = meshgen.kuhn_cube(m)
    return t.xyz, t.tets, meshgen.tet_centroids(t)


def _cell_meshes(ms, seed, contrast, radius, count):
    """Macro cells of ms[c]^3 hexahedra side by side along x, each with up to `count` ellipsoidal
    inclusions (semi-axes U(radius) in cell units) of Young's modulus `contrast`."""
    rng = np.random.default_rng(seed)
    h = 1.0 / 16.0
    xyz, tets, mat, box, no, to = [], [], [], [], [0], [0]
    for c, m in enumerate(ms):
        x, t, cen = _cell_template(m)
        inside = np.zeros(t.shape[0], bool)
        for _ in range(rng.integers(1, count + 1)):
            inside |= (((cen - rng.uniform(0, 1, 3)) / rng.uniform(*radius, 3)) ** 2).sum(1) < 1.0
        lo = np.array([c * h, 0.0, 0.0])
        xyz.append(lo + x * h)
        tets.append(t)
        mat.append(inside.astype(np.int32))
        box.append([lo[0], lo[0] + h, 0.0, h, 0.0, h])
        no.append(no[-1] + x.shape[0])
        to.append(to[-1] + t.shape[0])
    return meshgen.CellMeshes(node_off=np.array(no, np.int64), xyz=np.concatenate(xyz), tet_off=np.array(to, np.int64),
                              tets=np.concatenate(tets).astype(np.int32), mat=np.concatenate(mat), box=np.array(box),
                              E=np.array([1.0, contrast]), nu=np.array([0.3, 0.3]), m=np.array(ms, np.int32))


def _edges(case):
    e = [int(v) for v in case["edges"].split(",")]
    return [e[c % len(e)] for c in range(case["cells"])]


def _train_inputs(case, seed):
    """(voxel inputs [n, 4096], targets [n, 729, 24]): smooth moduli fields, small basis corrections."""
    g = _gen(seed)
    n = case["cells"]
    coarse = torch.rand((n, 1, 6, 6, 6), generator=g, device=DEV)
    vox = torch.nn.functional.interpolate(coarse, size=(16, 16, 16), mode="trilinear", align_corners=True)
    vox = (vox > 0.6).to(torch.float32).reshape(n, 4096)
    target = 0.2 * torch.randn((n, 729, 24), generator=g, device=DEV)
    return _host(vox), _host(target.to(torch.float32))


def _net_params(seed):
    """He-uniform weights as after a short training: every layer carries signal."""
    rng = np.random.default_rng(seed)
    parts = [rng.uniform(-1, 1, 27 * 32 * 4) * math.sqrt(6.0 / 108), rng.uniform(-0.1, 0.1, 32)]
    for layer in range(3):
        w = rng.uniform(-1, 1, (27, 32, 32)) * math.sqrt(6.0 / 864)
        b = rng.uniform(-0.1, 0.1, 32)
        if layer == 2:
            w *= 0.1
            w[:, 24:] = 0.0
            b[24:] = 0.0
        parts += [w.ravel(), b]
    return np.concatenate(parts).astype(np.float32)


# ------------------------------------------------------------------------------ prepare

def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, seed), kind=case["kind"])


def _precision(case):
    return {"fp64": fem.FP64, "fp32_ir": fem.FP32_IR}[case["precision"]]


def _prepare_potential(case, seed):
    xyz, tets, mat, sigma, nodes, values = _potential_inputs(case, seed)
    torch.cuda.synchronize()
    S = fem.System(fem.SCALAR, xyz, tets, mat)
    return {"system": S, "sigma": sigma, "nodes": nodes, "values": values, "precision": _precision(case),
            "x": torch.empty(S.n_rows, dtype=F64, device=DEV)}


def _prepare_potential_driver(case, seed):
    xyz, tets, mat, sigma, nodes, values = _potential_inputs(case, seed)
    mesh = meshgen.Mesh(xyz=_host(xyz), tets=_host(tets), mat=_host(mat), n=case["n"])
    return {"problem": meshgen.ScalarProblem(mesh, sigma, _host(nodes), _host(values)), "precision": _precision(case)}


def _prepare_elastic_driver(case, seed):
    xyz, tets, fixed, faces, load_ = _elastic_inputs(case["n"], case["jitter"], seed)
    mesh = meshgen.Mesh(xyz=_host(xyz), tets=_host(tets), mat=np.zeros(tets.shape[0], np.int32), n=case["n"])
    m = fixed.numel()
    return {"problem": meshgen.ElasticProblem(
        mesh=mesh, E=np.array([1.0]), nu=np.array([0.3]), bc_nodes=_host(fixed), bc_mask=np.full(m, 7, np.int32),
        bc_values=np.zeros((m, 3)), faces=_host(faces), face_elem=np.zeros(faces.shape[0], np.int32), traction=load_)}


def _prepare_product(case, seed):
    xyz, tets = _cube(case["n"], 0.1, seed)
    mat = _marked(xyz, tets, 40, 0.03, 0.1, seed)
    torch.cuda.synchronize()
    S = fem.System(fem.ELASTIC, xyz, tets, mat)
    S.assemble_elastic([1.0, 100.0], [0.3, 0.3])
    x = torch.randn(S.n_rows, generator=_gen(seed + 1), dtype=F64, device=DEV)
    return {"system": S, "x": x, "y": torch.empty_like(x)}


def _bases_inputs(case, seed):
    return _cell_meshes(_edges(case), seed, 10.0, (0.15, 0.45), 3)


def _prepare_bases(case, seed):
    cells = Cells(_bases_inputs(case, seed))
    return {"cells": cells, "bases": torch.empty((cells.n_nodes, 8, 3), dtype=F64, device=DEV)}


def _prepare_twolevel(case, seed):
    n = case["n"]
    xyz, tets, fixed, faces, load_ = _elastic_inputs(n, 0.0, seed)
    mat = _marked(xyz, tets, 2000, 0.015, 0.035, seed)
    E, nu = np.array([1.0, 10.0]), np.array([0.3, 0.3])
    dofs = (3 * fixed[:, None] + torch.arange(3, device=DEV, dtype=torch.int32)).reshape(-1).contiguous()
    zero = torch.zeros(dofs.numel(), dtype=F64, device=DEV)
    torch.cuda.synchronize()
    S, K = fem.System(fem.ELASTIC, xyz, tets, mat), fem.System(fem.ELASTIC, xyz, tets, mat)
    S.set_kuhn_grid(n)
    K.set_kuhn_grid(n)
    S.add_traction(_host(faces), load_)
    S.assemble_elastic(E, nu)
    K.assemble_elastic_textbook(E, nu)
    S.apply_dirichlet(dofs, zero)
    K.apply_dirichlet(dofs, zero)
    mesh = meshgen.Mesh(xyz=_host(xyz), tets=_host(tets), mat=_host(mat), n=n)
    cc = meshgen.cube_cells(mesh, E, nu, 8)
    cells = Cells(cc.cells)
    cells.build_bases(tol=1e-8)
    T = TwoLevel(S, cells, cc, _host(dofs))
    T.set_smoother(K, matrix_free=True)
    T.set_matrix_free(True)
    return {"solver": T, "system": S, "x0": torch.zeros(S.n_rows, dtype=F64, device=DEV),
            "x": torch.empty(S.n_rows, dtype=F64, device=DEV)}


def _cracked_inputs(case, seed):
    n = case["n"]
    xyz, tets = _cube(n, 0.0, seed)
    cracks = xfem.random_cracks(case["cracks"], 0.05, 0.15, 5)
    sigma = 0.5 + torch.rand(tets.shape[0], generator=_gen(seed), dtype=F64, device=DEV)
    node = torch.arange((n + 1) ** 3, device=DEV)
    plane = (n + 1) ** 2
    lo, hi = node[:plane], node[node >= plane * n]
    nodes = torch.cat([lo, hi]).to(torch.int32)
    values = torch.cat([torch.ones(lo.numel()), torch.zeros(hi.numel())]).to(DEV, F64)
    return xyz, tets, cracks, sigma, nodes, values


def _prepare_cracked(case, seed):
    xyz, tets, cracks, sigma, nodes, values = _cracked_inputs(case, seed)
    mesh = meshgen.Mesh(xyz=_host(xyz), tets=_host(tets), mat=np.zeros(tets.shape[0], np.int32), n=case["n"])
    return {"mesh": mesh, "cracks": cracks, "sigma": _host(sigma), "enrichment": xfem.enrich(mesh.xyz, mesh.tets, cracks),
            "nodes": _host(nodes), "values": _host(values)}


def _predict_inputs(case, seed):
    return _cell_meshes([8] * case["cells"], seed, 100.0, (0.24, 0.56), 4)


def _prepare_predict(case, seed):
    net = CoarseNet()
    net.set_params(_net_params(seed))
    cells = Cells(_predict_inputs(case, seed))
    return {"net": net, "cells": cells, "bases": torch.empty((cells.n_nodes, 8, 3), dtype=F64, device=DEV)}


def _prepare_gradient(case, seed):
    net = CoarseNet()
    net.set_params(_net_params(seed))
    vox, target = _train_inputs(case, seed)
    return {"net": net, "vox": vox, "target": target}


_PREPARE = {"potential": _prepare_potential, "potential_driver": _prepare_potential_driver,
            "elastic_driver": _prepare_elastic_driver, "product": _prepare_product, "bases": _prepare_bases,
            "twolevel": _prepare_twolevel, "cracked": _prepare_cracked, "predict": _prepare_predict,
            "gradient": _prepare_gradient}


# ------------------------------------------------------------------------------ run

def run(s):
    return _RUN[s["kind"]](s)


def _bases_of(s):
    check(load().msfem_cells_get_bases(s["cells"].h, C.c_void_p(s["bases"].data_ptr()), 1), "cells_get_bases")
    return s["bases"]


def _run_potential(s):
    S = s["system"]
    S.clear()
    S.assemble_scalar(s["sigma"])
    S.apply_dirichlet(s["nodes"], s["values"], fem.ROW_AND_COLUMN)
    S.copy_f_to_x()
    S.solve(fem.PCG_JACOBI, s["precision"], tol=1e-13)
    return S.get_x(s["x"])


def _run_potential_driver(s):
    return fem.fem_scalar_driver(s["problem"], fem.PCG_JACOBI, s["precision"], min_residual=1e-13)[0]


def _run_elastic_driver(s):
    return fem.fem_elastic_driver(s["problem"], fem.PCG_JACOBI, fem.FP64, min_residual=1e-12)[0]


def _run_product(s):
    check(load().msfem_spmv(s["system"].h, C.c_void_p(s["x"].data_ptr()), C.c_void_p(s["y"].data_ptr()), 1), "spmv")
    return s["y"]


def _run_bases(s):
    s["cells"].build_bases(fem.FP64, tol=1e-12)
    return _bases_of(s)


def _run_twolevel(s):
    s["system"].set_x(s["x0"])
    s["solver"].solve(tol=1e-11, precision=fem.FP64)
    return s["system"].get_x(s["x"])


def _run_cracked(s):
    S, _ = xfem.build_system(s["mesh"], s["cracks"], s["sigma"], s["enrichment"])
    S.apply_dirichlet(s["nodes"], s["values"], fem.ROW_AND_COLUMN)
    S.copy_f_to_x()
    S.solve(fem.GMRES, fem.FP32_IR, tol=1e-13, restart=50)
    x = S.get_x()
    S.close()
    return x


def _run_predict(s):
    s["net"].predict(s["cells"])
    return _bases_of(s)


def _run_gradient(s):
    loss, grad = s["net"].loss_grad(s["vox"], s["target"])
    return np.float32(loss), grad


_RUN = {"potential": _run_potential, "potential_driver": _run_potential_driver, "elastic_driver": _run_elastic_driver,
        "product": _run_product, "bases": _run_bases, "twolevel": _run_twolevel, "cracked": _run_cracked,
        "predict": _run_predict, "gradient": _run_gradient}


# ------------------------------------------------------------------------------ work

def work(case):
    """Inputs read once and outputs written once; for the solves the element matrices formed once and
    one product with the matrix (no iteration count is known beforehand)."""
    kind = case["kind"]
    if kind in ("predict", "gradient"):
        cells = case["cells"]
        conv = 2.0 * cells * 4096 * 27 * (4 * 32 + 2 * 32 * 32 + 32 * 24)
        if kind == "predict":
            return {"bytes": cells * (3072 * 4 + 729 * 24 * 8.0), "flops": conv}
        return {"bytes": cells * (4096 + 729 * 24) * 4.0, "flops": 3 * conv}
    if kind == "bases":
        nodes, tets = sum((m + 1) ** 3 for m in _edges(case)), sum(6 * m ** 3 for m in _edges(case))
        return {"bytes": nodes * (3 + 24) * 8.0 + tets * 20.0, "flops": tets * (300.0 + 8 * 288)}
    n = case["n"]
    nodes, tets = (n + 1.0) ** 3, 6.0 * n ** 3
    mesh = nodes * 24 + tets * 20
    if kind == "product":
        return {"bytes": (15 * nodes) * 76 + nodes * 48, "flops": 2 * 9 * 15 * nodes}
    if kind in ("elastic_driver", "twolevel"):
        return {"bytes": mesh + nodes * 24, "flops": tets * (300.0 + 288)}
    return {"bytes": mesh + nodes * 8, "flops": tets * (100.0 + 32)}


# ------------------------------------------------------------------------------ exact (plain torch, 64 bits)

def exact(case, seed):
    f = _EXACT.get(case["kind"])
    return f(case, seed) if f else None  # the two-level solve: 1e4 and more Krylov steps by any plain method


def _simplices(P):
    """P [e, k+1, 3]: gradients of the barycentric functions in the simplex's own span, and measures."""
    E = P[:, 1:] - P[:, :1]
    G = E @ E.transpose(1, 2)
    g = torch.linalg.inv(G) @ E
    g = torch.cat([-g.sum(1, keepdim=True), g], 1)
    return g, torch.linalg.det(G).sqrt() / [1, 1, 2, 6][P.shape[1] - 1]


def _elastic_blocks(P, E, nu):
    """[e, 3 k1, 3 k1] element matrices, block (I, J) = V (l gJ gI' + m gI gJ' + m gI.gJ 1)."""
    g, V = _simplices(P)
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    A = (V * lam)[:, None, None, None, None] * torch.einsum("eja,eib->eiajb", g, g)
    A += (V * mu)[:, None, None, None, None] * torch.einsum("eia,ejb->eiajb", g, g)
    gg = torch.einsum("eic,ejc->eij", g, g) * (V * mu)[:, None, None]
    A += gg[:, :, None, :, None] * torch.eye(3, dtype=F64, device=DEV)[None, None, :, None, :]
    k = 3 * P.shape[1]
    return A.reshape(-1, k, k)


def _dense(n, dofs, A):
    K = torch.zeros(n * n, dtype=F64, device=DEV)
    idx = (dofs[:, :, None] * n + dofs[:, None, :]).reshape(-1)
    K.index_add_(0, idx, A.reshape(-1))
    return K.reshape(n, n)


def _vector_dofs(elems):
    return (3 * elems.long()[:, :, None] + torch.arange(3, device=DEV)).reshape(elems.shape[0], -1)


def _apply(n, dofs, A, x):
    y = torch.zeros(n, dtype=F64, device=DEV)
    y.index_add_(0, dofs.reshape(-1), torch.einsum("eij,ej->ei", A, x[dofs]).reshape(-1))
    return y


def _cg(product, diag, b, free, tol=1e-14, most=20000):
    """Jacobi CG on the free unknowns, restarted on the true residual."""
    x = torch.zeros_like(b)
    b = torch.where(free, b, torch.zeros_like(b))
    goal = tol * b.norm()
    for _ in range(6):
        r = b - torch.where(free, product(x), torch.zeros_like(b))
        if r.norm() <= goal:
            break
        z = r / diag
        p, rz = z.clone(), torch.dot(r, z)
        for it in range(most):
            q = torch.where(free, product(p), torch.zeros_like(b))
            a = rz / torch.dot(p, q)
            x += a * p
            r -= a * q
            z = r / diag
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
            if it % 20 == 0 and r.norm() <= 0.5 * goal:
                break
    return x


def _scalar_solution(n, dofs, A, nodes, values):
    free = torch.ones(n, dtype=torch.bool, device=DEV)
    free[nodes.long()] = False
    g = torch.zeros(n, dtype=F64, device=DEV)
    g[nodes.long()] = values
    diag = torch.zeros(n, dtype=F64, device=DEV)
    diag.index_add_(0, dofs.reshape(-1), torch.diagonal(A, dim1=1, dim2=2).reshape(-1))
    x = _cg(lambda v: _apply(n, dofs, A, v), diag, -_apply(n, dofs, A, g), free)
    return torch.where(free, x, g)


def _exact_potential(case, seed):
    xyz, tets, mat, sigma, nodes, values = _potential_inputs(case, seed)
    g, V = _simplices(xyz[tets.long()])
    A = torch.einsum("eic,ejc->eij", g, g) * (V * torch.from_numpy(sigma).to(DEV)[mat.long()])[:, None, None]
    return _scalar_solution(xyz.shape[0], tets.long(), A, nodes, values)


def _exact_elastic_driver(case, seed):
    xyz, tets, fixed, faces, load_ = _elastic_inputs(case["n"], case["jitter"], seed)
    n = 3 * xyz.shape[0]
    one = torch.ones(tets.shape[0], dtype=F64, device=DEV)
    K = _dense(n, _vector_dofs(tets), _elastic_blocks(xyz[tets.long()], one, 0.3 * one))
    P = xyz[faces.long()]
    area = torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]).norm(dim=1) / 2
    F = torch.zeros(n, dtype=F64, device=DEV)
    per = (torch.from_numpy(load_).to(DEV) * area[:, None] / 3)[:, None, :].expand(-1, 3, -1)
    F.index_add_(0, _vector_dofs(faces).reshape(-1), per.reshape(-1))
    first = 3 * fixed.numel()  # the fixed nodes are the first ones
    x = torch.zeros(n, dtype=F64, device=DEV)
    x[first:] = torch.linalg.solve(K[first:, first:], F[first:])
    return x.cpu().numpy()


def _exact_product(case, seed):
    xyz, tets = _cube(case["n"], 0.1, seed)
    mat = _marked(xyz, tets, 40, 0.03, 0.1, seed)
    n = 3 * xyz.shape[0]
    x = torch.randn(n, generator=_gen(seed + 1), dtype=F64, device=DEV)
    E = torch.tensor([1.0, 100.0], dtype=F64, device=DEV)[mat.long()]
    return _apply(n, _vector_dofs(tets), _elastic_blocks(xyz[tets.long()], E, torch.full_like(E, 0.3)), x)


def _dirichlet(n, elems, A, fixed, X):
    """X [n, R, 3] with its free entries replaced by the solution of the zero-source problem."""
    K = _dense(3 * n, _vector_dofs(elems), A)
    free = (~fixed).repeat_interleave(3)
    Y = X.transpose(1, 2).reshape(3 * n, -1).clone()
    Y[free] = torch.linalg.solve(K[free][:, free], -K[free][:, ~free] @ Y[~free])
    return Y.reshape(n, 3, -1).transpose(1, 2)


def _cell_bases(m, xyz, tets, E):
    """[nodes, 8, 3] Order1 bases of one structured cell: linear on its edges, the face problems on
    material 0, the volume problems with the cell's own moduli."""
    n = (m + 1) ** 3
    node = torch.arange(n, device=DEV)
    ijk = torch.stack([node % (m + 1), node // (m + 1) % (m + 1), node // (m + 1) ** 2], 1)
    at = [(ijk[:, a] == side * m) for a in range(3) for side in range(2)]
    hats = [[1 - t, t] for t in (ijk.to(F64) / m).unbind(1)]
    X = torch.zeros((n, 8, 3), dtype=F64, device=DEV)
    edge = sum(f.int() for f in at) >= 2
    for v in range(8):
        X[:, v] = (hats[0][v & 1] * hats[1][v >> 1 & 1] * hats[2][v >> 2])[:, None]
    for f in at:
        nodes = node[f]
        on = f[tets]
        hit = on.sum(1) == 3
        local = torch.full((n,), -1, device=DEV)
        local[nodes] = torch.arange(nodes.numel(), device=DEV)
        tri = local[tets[hit][on[hit]].reshape(-1, 3)]
        one = torch.ones(tri.shape[0], dtype=F64, device=DEV)
        A = _elastic_blocks(xyz[nodes][tri], one, 0.3 * one)
        X[nodes] = _dirichlet(nodes.numel(), tri, A, edge[nodes], X[nodes])
    return _dirichlet(n, tets, _elastic_blocks(xyz[tets], E, torch.full_like(E, 0.3)), sum(f.int() for f in at) > 0, X)


def _exact_bases(case, seed):
    cm = _bases_inputs(case, seed)
    E = torch.from_numpy(cm.E).to(DEV)
    out = []
    for c in range(cm.n_cells):
        xyz, tets, mat, _ = cm.cell(c)
        out.append(_cell_bases(int(cm.m[c]), torch.from_numpy(xyz).to(DEV), torch.from_numpy(tets).to(DEV).long(),
                               E[torch.from_numpy(mat).to(DEV).long()]))
    return torch.cat(out)


def _volume(a, b, c, d):
    return torch.det(torch.stack([b - a, c - a, d - a], 1)).abs() / 6


def _positive_volume(P, d):
    """Volume of {linear function with vertex values d >= 0} in each tetrahedron P."""
    order = torch.argsort(d, dim=1, descending=True)
    P, d = torch.gather(P, 1, order[:, :, None].expand(-1, -1, 3)), torch.gather(d, 1, order)

    def x(a, b):
        return P[:, a] + (d[:, a] / (d[:, a] - d[:, b]))[:, None] * (P[:, b] - P[:, a])
    full = _volume(P[:, 0], P[:, 1], P[:, 2], P[:, 3])
    one = _volume(P[:, 0], x(0, 1), x(0, 2), x(0, 3))
    three = full - _volume(P[:, 3], x(0, 3), x(1, 3), x(2, 3))
    ac, ae, bc, be = x(0, 2), x(0, 3), x(1, 2), x(1, 3)
    two = _volume(P[:, 0], ac, ae, P[:, 1]) + _volume(P[:, 1], ac, ae, be) + _volume(P[:, 1], ac, be, bc)
    k = (d >= 0).sum(1)
    return torch.where(k == 1, one, torch.where(k == 2, two, three))


def _exact_cracked(case, seed):
    xyz, tets, cracks, sigma, nodes, values = _cracked_inputs(case, seed)
    t = tets.long()
    n = xyz.shape[0]
    cen, nor = (torch.from_numpy(a).to(DEV) for a in (cracks.centre, cracks.normal))
    P = xyz[t]
    mid = P.mean(1)
    of = torch.full((t.shape[0],), -1, device=DEV)
    for k in range(cen.shape[0] - 1, -1, -1):  # the lowest-numbered crack wins
        d = (P - cen[k]) @ nor[k]
        rel = mid - cen[k]
        flat = rel - (rel @ nor[k])[:, None] * nor[k]
        cut = (d.max(1).values > 0) & (d.min(1).values < 0) & ((flat ** 2).sum(1) < cracks.radius[k] ** 2)
        of[cut] = k
    g, V = _simplices(P)
    K = torch.einsum("eic,ejc->eij", g, g) * sigma[:, None, None]
    hit = of >= 0
    Pc, Kc, k = P[hit], K[hit], of[hit]
    d = torch.einsum("evc,ec->ev", Pc - cen[k][:, None], nor[k])
    plus = _positive_volume(Pc, d)
    minus = V[hit] - plus
    H = torch.where(d >= 0, 1.0, -1.0).to(F64)
    pairs, inv = torch.unique((k[:, None] * n + t[hit]).reshape(-1), return_inverse=True)
    total = n + pairs.numel()
    up, down = 1 - H, -1 - H
    w = torch.zeros((Kc.shape[0], 8, 8), dtype=F64, device=DEV)
    basis_up, basis_down = torch.cat([torch.ones_like(H), up], 1), torch.cat([torch.ones_like(H), down], 1)
    w += plus[:, None, None] * basis_up[:, :, None] * basis_up[:, None, :]
    w += minus[:, None, None] * basis_down[:, :, None] * basis_down[:, None, :]
    cutA = w * Kc.repeat(1, 2, 2)
    cut_dofs = torch.cat([t[hit], n + inv.reshape(-1, 4)], 1)
    rest, restA = t[~hit], K[~hit] * V[~hit][:, None, None]
    rows = torch.cat([rest.repeat_interleave(4, 1).reshape(-1), cut_dofs.repeat_interleave(8, 1).reshape(-1)])
    cols = torch.cat([rest.repeat(1, 4).reshape(-1), cut_dofs.repeat(1, 8).reshape(-1)])
    S = torch.sparse_coo_tensor(torch.stack([rows, cols]), torch.cat([restA.reshape(-1), cutA.reshape(-1)]),
                                (total, total)).coalesce()
    i, v = S.indices(), S.values()
    diag = torch.zeros(total, dtype=F64, device=DEV).index_add_(0, i[0][i[0] == i[1]], v[i[0] == i[1]])
    S = S.to_sparse_csr()
    free = torch.ones(total, dtype=torch.bool, device=DEV)
    free[nodes.long()] = False
    fixed = torch.zeros(total, dtype=F64, device=DEV)
    fixed[nodes.long()] = values
    x = _cg(lambda y: S @ y, diag, -(S @ fixed), free)
    return torch.where(free, x, fixed).cpu().numpy()


class _Net:
    """The network in 64 bits: parameters as leaves, voxel fields to node corrections."""

    def __init__(self, params, grad):
        self.flat = torch.from_numpy(params).to(DEV, F64).requires_grad_(grad)
        self.layers, at = [], 0
        for cin in (4, 32, 32, 32):
            w = self.flat[at:at + 27 * 32 * cin].reshape(3, 3, 3, 32, cin).permute(3, 4, 0, 1, 2)
            at += 27 * 32 * cin
            self.layers.append((w, self.flat[at:at + 32]))
            at += 32
        i = torch.arange(16, device=DEV)
        c = (2.0 * i.to(F64) + 1.0) / 16 - 1.0
        z, y, x = torch.meshgrid(c, c, c, indexing="ij")
        self.coords = torch.stack([x, y, z])
        self.node = (i + 1) >> 1
        self.count = torch.bincount(self.node).to(F64)

    def corrections(self, vox):
        """[n, 4096] -> [n, 729, 24]."""
        n = vox.shape[0]
        a = torch.cat([vox.reshape(n, 1, 16, 16, 16), self.coords.expand(n, -1, -1, -1, -1)], 1)
        for k, (w, b) in enumerate(self.layers):
            a = torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1))
            a = a.unfold(2, 3, 1).unfold(3, 3, 1).unfold(4, 3, 1)  # [n, ci, z, y, x, dz, dy, dx]
            a = torch.einsum("nizyxabc,oiabc->nozyx", a, w) + b.reshape(1, -1, 1, 1, 1)
            if k < 3:
                a = a.relu()
        a = a[:, :24]
        for dim in (2, 3, 4):
            s = torch.zeros([9 if d == dim else a.shape[d] for d in range(5)], dtype=F64, device=DEV)
            shape = [1] * 5
            shape[dim] = 9
            a = s.index_add(dim, self.node, a) / self.count.reshape(shape)
        keep = torch.ones((9, 9, 9), dtype=F64, device=DEV)
        keep[::8, ::8, ::8] = 0.0
        return (a * keep).permute(0, 2, 3, 4, 1).reshape(n, 729, 24)


def _trilinear():
    t = torch.arange(9, device=DEV, dtype=F64) / 8
    z, y, x = (a.reshape(-1) for a in torch.meshgrid(t, t, t, indexing="ij"))
    f = [(x if v & 1 else 1 - x) * (y if v >> 1 & 1 else 1 - y) * (z if v >> 2 else 1 - z) for v in range(8)]
    return torch.stack(f, 1).repeat_interleave(3, 1)


def _exact_predict(case, seed):
    cm = _predict_inputs(case, seed)
    n = cm.n_cells
    value = torch.from_numpy(np.log(cm.E) / math.log(100.0)).to(DEV)[torch.from_numpy(cm.mat).to(DEV).long()]
    value = value.reshape(n, 8, 8, 8, 6)
    octant = torch.arange(8, device=DEV)
    half = torch.stack([octant & 1, octant >> 1 & 1, octant >> 2], 1)
    orders = [(0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)]
    ok = torch.stack([(half[:, o[0]] >= half[:, o[1]]) & (half[:, o[1]] >= half[:, o[2]]) for o in orders], 1).to(F64)
    v = torch.einsum("nzyxt,ot->nzyxo", value, ok / ok.sum(1, keepdim=True))
    v = v.reshape(n, 8, 8, 8, 2, 2, 2).permute(0, 1, 4, 2, 5, 3, 6).reshape(n, 4096)
    net = _Net(_net_params(seed), False)
    out = [net.corrections(v[c:c + 8]) for c in range(0, n, 8)]
    return (torch.cat(out) + _trilinear()).reshape(-1, 8, 3)


def _exact_gradient(case, seed):
    vox, target = (torch.from_numpy(a).to(DEV, F64) for a in _train_inputs(case, seed))
    net = _Net(_net_params(seed), True)
    loss = torch.zeros((), dtype=F64, device=DEV)
    for c in range(0, vox.shape[0], 8):
        part = ((net.corrections(vox[c:c + 8]) - target[c:c + 8]) ** 2).sum() / target.numel()
        part.backward()
        loss += part.detach()
    return loss.item(), net.flat.grad.cpu().numpy()


_EXACT = {"potential": _exact_potential, "potential_driver": lambda c, s: _exact_potential(c, s).cpu().numpy(),
          "elastic_driver": _exact_elastic_driver, "product": _exact_product, "bases": _exact_bases,
          "cracked": _exact_cracked, "predict": _exact_predict, "gradient": _exact_gradient}
