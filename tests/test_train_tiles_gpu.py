"""The fused gradient pass (k_train, csrc/nn_flux.cu) where its grid changes: a single row tile of 128, 37
blocks of four tiles (148 tiles, a multiple of 512 rows), 149 splits of one tile on 148 blocks, and a ragged
third round of them.  The order of its sums is held in test_train_sums_gpu.py.  Tolerance here: the
2e-3 relative L2 per layer of the gradient tests (BF16 operands, FP32 sums); the loss to 1e-3."""
import numpy as np
import pytest

from test_nn_gpu import FluxNet, layer_slices, mo, random_params, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [1, 148, 149, 301])
def test_gradient_at_tile_counts(tiles):
    rng = np.random.default_rng(tiles)
    with FluxNet() as net:
        p = random_params(net, 12)
        x = rng.normal(0, 1, (128 * tiles, 17)).astype(np.float32)
        t = rng.normal(0, 1, (128 * tiles, 8)).astype(np.float32)
        loss, g = net.gradients(x, t)
        lo, go = mo.loss_and_grad(p, x.astype(np.float64), t.astype(np.float64), shp=net.shapes)
        assert abs(loss - lo) <= 1e-3 * lo
        for s in layer_slices(net):
            assert rel(g[s], go[s]) < 2e-3, (s, rel(g[s], go[s]))
