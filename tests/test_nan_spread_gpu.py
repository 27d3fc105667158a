"""An invalid state in FP32: one step from a state with a NaN in one cell makes every value NaN that the FP64
path (the reference's arithmetic) makes NaN.  The limiters and the wave-speed bounds of the FP32 kernels use
one-instruction minima and maxima; those that drop a NaN would leave the cells around it looking valid.  Rows
of even and of odd length take different Riemann kernels; in the supersonic flow an edge's EMF is the plain
one of its upwind corner, which only the bounds connect with the other three."""
import numpy as np
import pytest

from dumses_hybrid_b200 import Context, Params, condinit

pytestmark = pytest.mark.gpu


def after_step(p, bad, dt):
    with Context(p) as g:
        g.upload(bad)
        g.boundary(0.0, 0.0)
        g.godunov(dt, 0.0)
        act = tuple(slice(3, 3 + n) for n in (p.nx, p.ny, p.nz))
        return np.isnan(g.download()[act][..., :8])


@pytest.mark.parametrize("variable", [0, 1, 4, 6])
@pytest.mark.parametrize("speed", [0.0, 30.0])
@pytest.mark.parametrize("nx", [16, 17])
def test_one_step_from_a_nan(nx, speed, variable):
    box = dict(ndim=3, nx=nx, ny=12, nz=11, xmin=0, xmax=1, ymin=0, ymax=1, zmin=0, zmax=1, courant=0.4)
    good = condinit(Params(**box), "orszag_tang")
    for v in (1, 2, 3):
        good[..., v] += speed * good[..., 0]
    good[..., 4] += 0.5 * good[..., 0] * 3 * speed**2 + speed * (good[..., 1] + good[..., 2])
    bad = good.copy(order="F")
    bad[3 + 8, 3 + 6, 3 + 5, variable] = np.nan
    dt = 1e-4
    want = after_step(Params(**box), bad, dt)
    got = after_step(Params(precision="fp32", **box), bad, dt)
    assert want.any()
    missed = want & ~got
    assert not missed.any(), (int(missed.sum()), int(want.sum()), int(got.sum()), np.argwhere(missed)[:4].tolist())
