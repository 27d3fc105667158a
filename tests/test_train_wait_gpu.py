"""A wait of the one-kernel gradient pass (k_train, csrc/nn_flux.cu) that runs out: the products in flight
are still waited for, the block leaves without a step, the parameters keep their values, the call and the
network's later ones report DG_ERR_STATE, and the device stays usable.  A bound of zero makes every wait run
out; nothing hangs or faults."""
import time

import numpy as np
import pytest

import dumses_hybrid_b200 as dg
from test_nn_gpu import FluxNet, random_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [128, 512 * 149])
def test_pass_whose_wait_runs_out(rows):
    rng = np.random.default_rng(rows)
    x = rng.normal(0, 1, (rows, 17)).astype(np.float32)
    t = rng.normal(0, 1, (rows, 8)).astype(np.float32)
    with FluxNet() as net:
        if net.shape[0] > 64:
            pytest.skip("networks wider than 64 train by the kernel chain")
        random_params(net, 12)
        net.set_samples(x, t)
        want = net.gradients(x, t)
        net.train(1, batch=rows)
        kept = net.params()
        assert net.lib.dg_nn_wait_bound(net.h, 0.0) == dg.DG_OK
        t0 = time.monotonic()
        for call in (lambda: net.train(3, batch=rows), lambda: net.gradients(x, t), lambda: net.train(3, batch=rows)):
            with pytest.raises(dg.DumsesError) as e:
                call()
            assert e.value.code == -5  # DG_ERR_STATE
        assert time.monotonic() - t0 < 0.5  # no wait lasted its second
        assert np.array_equal(net.params(), kept)
    with FluxNet() as net:
        random_params(net, 12)
        again = net.gradients(x, t)
        assert again[0] == want[0] and np.array_equal(again[1], want[1])


def test_bounds_outside_the_range_are_refused():
    with FluxNet() as net:
        for s in (-1.0, float("nan"), 61.0):
            assert net.lib.dg_nn_wait_bound(net.h, s) == -1  # DG_ERR_ARG
        assert net.lib.dg_nn_wait_bound(None, 1.0) == -1
