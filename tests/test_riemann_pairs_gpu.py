"""The FP32 Riemann solves two cells per thread (csrc/riemann32.cuh, an even nx) and one cell per thread
(an odd nx) on either side of the rule, at the smallest rows and across a block's end: the face fluxes and
edge EMFs of one step against those of the bit-exact FP64 path.  Tolerance: a flux goes through fewer than a
thousand FP32 operations of 6e-8 each on this smooth start, so 1e-4 of the array's largest entry; a
neighbour read or a record written one place off is wrong by the flow's variation per cell, 1e-1."""
import numpy as np
import pytest

from dumses_hybrid_b200 import Context, Params, condinit

pytestmark = pytest.mark.gpu


def arrays(p, u0):
    F = (p.nx + 1) * (p.ny + 1) * (p.nz + 1)
    shape = (p.nz + 1, p.ny + 1, p.nx + 1)
    with Context(p) as g:
        g.upload(u0)
        g.boundary(0.0, 0.0)
        g.godunov(1e-3, 0.0)
        flux = [g.debug_array(d, 6 * F).reshape(shape + (6,)) for d in range(3)]
        emf = [g.debug_array(3 + d, F).reshape(shape) for d in range(3)]
    out = []
    for d in range(3):  # the records the step fills: one face more along d, one edge more across d
        out.append(flux[d][tuple(slice(0, n + (a == d)) for a, n in zip((2, 1, 0), (p.nz, p.ny, p.nx)))])
        out.append(emf[d][tuple(slice(0, n + (a != d)) for a, n in zip((2, 1, 0), (p.nz, p.ny, p.nx)))])
    return out


@pytest.mark.parametrize("iso", [False, True])
@pytest.mark.parametrize("nx,ny,nz", [(6, 7, 5), (7, 6, 5), (34, 5, 9), (35, 5, 9), (64, 17, 6), (62, 16, 8)])
def test_rows_of_either_parity(nx, ny, nz, iso):
    kw = dict(iso=1, ciso=1.0) if iso else {}
    box = dict(ndim=3, nx=nx, ny=ny, nz=nz, xmin=0, xmax=1, ymin=0, ymax=1, zmin=0, zmax=1, courant=0.4, **kw)
    p64, p32 = Params(**box), Params(precision="fp32", **box)
    u0 = condinit(p64, "orszag_tang")
    wave = 0.1 * np.sin(2 * np.pi * (np.arange(nz + 6) + 0.3) / nz)[None, None, :]
    u0[..., 3] += u0[..., 0] * wave
    u0[..., 1] += u0[..., 0] * wave
    for got, want in zip(arrays(p32, u0), arrays(p64, u0)):
        assert np.abs(want).max() > 0
        assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
