"""msfem_spmv and msfem_spmv_scaled32 on every kind of vector: device memory is used in place, host
memory and overlapping vectors go through copies; the values are the same bits."""
import ctypes as C

import numpy as np
import pytest
import torch

from multiscalefemsolver3d_b200 import fem, meshgen
from multiscalefemsolver3d_b200._lib import check, load

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(fem.SCALAR, 9), (fem.ELASTIC, 9), (fem.ELASTIC, 62)],
                ids=["scalar", "blocks", "blocks-two-rounds"])
def system(cuda, request):
    kind, n = request.param
    m = meshgen.cube_elastic(n=n, jitter=0.05, n_spheres=3, contrast=10.0, rmin=0.1, rmax=0.2).mesh
    S = fem.System(kind, m.xyz, m.tets, m.mat)
    if kind == fem.SCALAR:
        S.assemble_scalar([1.0, 10.0])
    else:
        S.assemble_elastic([1.0, 10.0], [0.3, 0.3])
    return S


@pytest.mark.parametrize("single", [False, True], ids=["fp64", "scaled-fp32"])
def test_vectors_of_every_kind(system, single):
    S, n = system, system.n_rows
    fn = load().msfem_spmv_scaled32 if single else load().msfem_spmv
    dt, tdt = (np.float32, torch.float32) if single else (np.float64, torch.float64)
    x = np.random.default_rng(1).standard_normal(n).astype(dt)
    ref = S.spmv_scaled32(x) if single else S.spmv(x)

    def call(px, py):
        check(fn(S.h, C.c_void_p(px), C.c_void_p(py), 1), "product")

    dx = torch.from_numpy(x).cuda()
    for off in (0, 1, 3):  # element offsets: no alignment beyond the type's
        buf, out = torch.zeros(n + 3, dtype=tdt, device="cuda"), torch.full((n + 6,), 7.0, dtype=tdt, device="cuda")
        buf[off:off + n] = dx
        torch.cuda.synchronize()
        call(buf[off:].data_ptr(), out[off:].data_ptr())
        np.testing.assert_array_equal(out[off:off + n].cpu().numpy(), ref)
        assert torch.all(out[:off] == 7) and torch.all(out[off + n:] == 7)
    y = np.empty(n, dt)
    call(dx.data_ptr(), y.ctypes.data)  # device to host
    np.testing.assert_array_equal(y, ref)
    dy = torch.empty(n, dtype=tdt, device="cuda")
    call(x.ctypes.data, dy.data_ptr())  # host to device
    np.testing.assert_array_equal(dy.cpu().numpy(), ref)
    for shift in (0, 5, n // 2):  # y over x, and over a part of it from either side
        for xo, yo in ((0, shift), (shift, 0)):
            buf = torch.zeros(n + shift, dtype=tdt, device="cuda")
            buf[xo:xo + n] = dx
            torch.cuda.synchronize()
            call(buf[xo:].data_ptr(), buf[yo:].data_ptr())
            np.testing.assert_array_equal(buf[yo:yo + n].cpu().numpy(), ref)


def test_product_against_the_stored_matrix(system):
    A = system.export_csr().to_scipy()
    x = np.random.default_rng(2).standard_normal(system.n_rows)
    y = system.spmv(x)
    # rounding of a row's sum: at most 45 (15 scalar) terms
    bound = 64 * np.finfo(np.float64).eps * (abs(A) @ np.abs(x))
    assert np.all(np.abs(y - A @ x) <= bound)
