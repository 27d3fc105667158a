"""The order of the FP32 sums behind a network gradient (k_train and k_adam, csrc/nn_flux.cu): a weight's
gradient is accumulated over 512 consecutive rows (128 where 512 does not divide the batch) and those
partials are added in order; a bias's gradient and the loss are summed per 128-row tile and added in tile
order.  A training run repeats only as far as this order does: the rounding of the weights to BF16 turns
a last bit of a gradient into 1e-5 of the loss a few steps later.

The gradient of the mean over 2^m rows is exactly 2^-k times that over 2^(m-k) rows (a power of two scales
every operand of the products without rounding), so the order is held without any tolerance: the gradient
of a batch is the in-order FP32 sum of its pieces' gradients, scaled, bit for bit."""
import numpy as np
import pytest

from test_nn_gpu import FluxNet, layer_slices, random_params

pytestmark = pytest.mark.gpu


def batch(rows, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(0, 1, (rows, 17)).astype(np.float32), rng.normal(0, 1, (rows, 8)).astype(np.float32)


def in_order(net, x, t, piece):
    """The gradients of x's pieces, each times piece / rows, added in FP32 in the order of the rows."""
    rows = x.shape[0]
    total = np.zeros(net.param_count, np.float32)
    for a in range(0, rows, piece):
        total += net.gradients(x[a:a + piece], t[a:a + piece])[1] * np.float32(piece / rows)
    return total


# 2 splits of one tile; 2 and 32 splits of four tiles; 256 splits, more than the chip's 148 blocks
@pytest.mark.parametrize("rows,piece", [(256, 128), (1024, 512), (16384, 512), (131072, 512)])
def test_gradient_is_the_ordered_sum_of_its_splits(rows, piece):
    x, t = batch(rows, rows)
    with FluxNet() as net:
        random_params(net, 12)
        got = net.gradients(x, t)[1]
        weights, biases = in_order(net, x, t, piece), in_order(net, x, t, 128)
        for n, s in enumerate(layer_slices(net)):  # weights and biases in turn
            want = biases if n % 2 else weights
            assert np.array_equal(got[s], want[s]), (n, np.abs(got[s] - want[s]).max())


@pytest.mark.parametrize("rows", [1024, 128 * 149, 128 * 301, 512 * 149])
def test_a_pass_repeats_its_bits(rows):
    x, t = batch(rows, 3)
    with FluxNet() as net:
        random_params(net, 12)
        loss, first = net.gradients(x, t)
        for _ in range(20):
            again, g = net.gradients(x, t)
            assert again == loss and np.array_equal(g, first)


def test_gradients_of_batches_in_any_order():
    """A batch of more, smaller splits than an earlier and larger one holds its own partials."""
    with FluxNet() as net:
        random_params(net, 12)
        x, t = batch(65536, 5)
        want = [net.gradients(x[:n], t[:n])[1] for n in (384, 65408)]
    with FluxNet() as net:
        random_params(net, 12)
        net.gradients(x, t)
        assert np.array_equal(net.gradients(x[:65408], t[:65408])[1], want[1])
        assert np.array_equal(net.gradients(x[:384], t[:384])[1], want[0])
