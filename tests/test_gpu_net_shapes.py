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


@pytest.mark.parametrize("n", [1, 3, 19])
def test_gradient_matches_the_oracle(cuda, n):
    """Loss and every layer's gradient against the oracle (64 bits, the network's BF16 points) over
    partials of one unit a block and of one or two; the bars of the two-cell test: BF16 values that fall on the
    other side of a rounding boundary cost up to 2e-3 of a layer's gradient."""
    net = _net(3)
    p = on.init_params(3)
    vox, tgt = _inputs(n, 40 + n)
    loss, g = net.loss_grad(vox, tgt)
    loss_ref, g_ref = on.loss_grad(p, vox, tgt)
    assert loss == pytest.approx(loss_ref, rel=1e-4)
    for lo, hi in [(0, on.L1), (on.layer_base(1), on.layer_base(2)), (on.layer_base(2), on.layer_base(3)),
                   (on.layer_base(3), on.PARAMS)]:
        assert np.linalg.norm(g[lo:hi] - g_ref[lo:hi]) <= 2e-3 * np.linalg.norm(g_ref[lo:hi])


@pytest.mark.parametrize("n", [320, 1280])
def test_gradient_of_a_batch_is_the_mean_of_its_eighths(cuda, n):
    """Ranges long enough for partial sums to be put away on the way (8 units of the 32-channel layers, 64 of
    the first).  A factor of eight in the norm is exact in every rounding, so batch and eighths have the same
    terms and differ by the FP32 order of their sums: 1e-4, as between two kernels of one pass."""
    net = _net(5)
    vox, tgt = _inputs(n, n)
    loss, g = net.loss_grad(vox, tgt)
    parts = [net.loss_grad(vox[k::8].copy(), tgt[k::8].copy()) for k in range(8)]
    assert loss == pytest.approx(np.mean([l for l, _ in parts]), rel=1e-5)
    ref = np.mean([q for _, q in parts], axis=0, dtype=np.float64)
    for lo, hi in [(0, on.L1), (on.layer_base(1), on.layer_base(2)), (on.layer_base(2), on.layer_base(3)),
                   (on.layer_base(3), on.PARAMS)]:
        assert np.linalg.norm(g[lo:hi] - ref[lo:hi]) <= 1e-4 * np.linalg.norm(ref[lo:hi])


@pytest.mark.parametrize("n", [1, 2, 38])
def test_forward_matches_the_oracle(cuda, n):
    """The first layer's ranges of plane pairs (fewer than two a multiprocessor, and more) through to the
    output, cell by cell at the bar of the few-cell test (BF16 rounding boundaries)."""
    net = _net(9)
    vox, _ = _inputs(n, 70 + n)
    vox *= np.linspace(0.2, 3.0, 16, dtype=np.float32).repeat(256)  # no two planes alike
    out = net.forward(vox)
    for k in sorted({0, n // 2, n - 1}):
        ref = on.forward(on.init_params(9), vox[k:k + 1])[0][1]
        assert np.linalg.norm(out[k] - ref) <= 5e-3 * np.linalg.norm(ref), k


@pytest.mark.parametrize("n", [1, 2, 9, 10, 19, 37, 38, 301])
def test_stacked_taps_give_the_bits_of_the_cell_kernel(cuda, n):
    """The default path (k_conv32_st: three z-taps an instruction, rings of planes and of accumulators,
    ranges of output planes cut anywhere in a cell) against the tcgen05 kernel that takes a cell a block.
    The products of each sum are added in one order, so all bits agree: ranges of one plane (n <= 9), of one
    or two, ranges that end on every plane of a cell (19, 37, 38), and long ones that go round both rings."""
    net, ref = _net(13), _net(13)
    ref.set_tensor_path(1)
    vox, tgt = _inputs(n, 100 + n)
    np.testing.assert_array_equal(net.forward(vox), ref.forward(vox))
    (loss, g), (l_ref, g_ref) = net.loss_grad(vox, tgt), ref.loss_grad(vox, tgt)
    assert loss == l_ref
    np.testing.assert_array_equal(g, g_ref)


def test_default_path_is_repeatable_from_two_threads(cuda):
    """Two networks on two threads: their kernels take whole multiprocessors (all of the tensor memory) in
    turn."""
    import threading
    vox, _ = _inputs(200, 1)
    nets = [_net(1), _net(2)]
    ref = [net.forward(vox) for net in nets]
    got = [None, None]

    def work(k):
        for _ in range(4):
            got[k] = nets[k].forward(vox)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=60)
    for k in range(2):
        np.testing.assert_array_equal(got[k], ref[k])
