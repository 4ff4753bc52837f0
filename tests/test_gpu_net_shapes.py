"""The network's kernels (csrc/neural.cu) at the batch sizes where their division of the work changes:
one cell, fewer steps than multiprocessors, one more than that, two per multiprocessor, ranges that
cross several cells."""
import numpy as np
import pytest

from multiscalefemsolver3d_b200.learned import CoarseNet
from oracle import neural as on

pytestmark = pytest.mark.gpu


def _net(seed):
    net = CoarseNet()
    net.set_params(on.init_params(seed))
    return net


def _inputs(n, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(0.0, 1.0, (n, 4096)).astype(np.float32), rng.normal(0.0, 0.05, (n, 729, 24)).astype(np.float32)


@pytest.mark.parametrize("n", [1, 2, 18, 19, 37, 38, 301])
def test_conv_ring_gives_the_bits_of_the_cell_kernel(cuda, n):
    """k_conv32's ring of planes over a range of cells against the tcgen05 kernel, which takes a cell a
    block: both sum the 54 k16 products in one order, so forward, loss and gradients are bit-equal."""
    net = _net(11)
    vox, tgt = _inputs(n, n)
    net.set_tensor_path(1)
    o_ref, (l_ref, g_ref) = net.forward(vox), net.loss_grad(vox, tgt)
    net.set_tensor_path(0)
    np.testing.assert_array_equal(net.forward(vox), o_ref)
    loss, g = net.loss_grad(vox, tgt)
    assert loss == l_ref
    np.testing.assert_array_equal(g, g_ref)
