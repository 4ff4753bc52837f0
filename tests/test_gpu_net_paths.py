"""Choosing the network's tensor-core path: the default has a number, so that a network on which another path was
chosen can return to it, with the same bits as one that never left it; numbers without a path are refused."""
import numpy as np
import pytest

from multiscalefemsolver3d_b200._lib import MsfemError
from multiscalefemsolver3d_b200.learned import CoarseNet
from oracle import neural as on

pytestmark = pytest.mark.gpu


def test_back_to_the_default_path(lib, cuda):
    rng = np.random.default_rng(11)
    vox = rng.normal(0.0, 1.0, (5, 4096)).astype(np.float32)
    tgt = rng.normal(0.0, 0.05, (5, 729, 24)).astype(np.float32)
    net = CoarseNet()
    net.set_params(on.init_params(3))
    out = net.forward(vox)
    loss, grad = net.loss_grad(vox, tgt)
    net.set_tensor_path(0)
    net.forward(vox)
    net.set_tensor_path(4)
    np.testing.assert_array_equal(net.forward(vox), out)
    loss4, grad4 = net.loss_grad(vox, tgt)
    assert loss4 == loss
    np.testing.assert_array_equal(grad4, grad)


@pytest.mark.parametrize("path", [-1, 5])
def test_unknown_paths_are_refused(lib, cuda, path):
    net = CoarseNet()
    with pytest.raises(MsfemError):
        net.set_tensor_path(path)
