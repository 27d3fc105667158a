"""FARGO's two segment lengths (fargo_short, csrc/step_impl.cuh): 16 rows of y per thread on large grids, 4
where those would leave the chip idle, chosen apart for the EMFs and for the remap.  One update on grids that
take 16 rows for both, and for the remap alone: last segments of 1 to 16 rows, lines shorter than a thread's
window of 19 rows (which then wraps several times), and shifts of whole cells, of fractions of several cells
and of more cells than a segment has rows.

FP64 against the oracle, bit for bit.  FP32 against FP64: the remap is the donor cell's value plus an FP32
increment and the fields are moved by FP32 sums over at most 20 cells, so 20 x 6e-8 x a few = 1e-5 of an
array's largest value; a row read or written one place off is wrong by this random state's variation, 1e-1.
The bounds-checked build then repeats every grid in both precisions: no access outside the buffers."""
import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

import dumses_hybrid_b200 as dg
from dumses_hybrid_b200 import Context, Params
from test_parity_large_gpu import fargo_pair, fargo_state_for, shifts

pytestmark = pytest.mark.gpu

HERE = pathlib.Path(__file__).resolve().parent
NX = 20  # cell centres x = (2 i - 21) / 40
# ny, nz, dt, long EMFs
GRIDS = {
    "whole cells, 10 rows in the last segment": (41, 1900, 40 / 96, True),  # 1, 3, .. 19 cells
    "fractions of several cells": (41, 1900, 0.33, True),
    "17 faces, 1 row in the last segment": (16, 2800, 0.3, True),
    "16 faces, one whole segment": (15, 5500, 0.3, True),
    "6 faces, the window wraps": (5, 5500, 0.1, True),
    "4 faces, the fewest": (3, 5500, 0.05, True),
    "16 rows for the remap alone": (41, 900, 0.4, False),
}


def params(ny, nz, precision="fp64"):
    return Params(ndim=3, iso=1, nx=NX, ny=ny, nz=nz, xmin=-0.5, xmax=0.5, ymin=0.0, ymax=ny / 64, zmin=0.0, zmax=nz / 64,
                  gamma=5 / 3, ciso=1.0, omega0=1.0, courant=0.8, bdtypex="shearingbox", fargo=True, precision=precision)


def takes_long(p, waves):
    return (p.nx + 1) * (p.nz + 1) * ((p.ny + 1 + 15) // 16) >= waves * 148 * 3 * 128


def updated(p, u0, dt):
    with Context(p) as g:
        g.upload(u0)
        g.boundary(0.0, 0.0)
        g.fargo_update(dt)
        g.boundary(0.0, dt)
        return g.download()


@pytest.mark.parametrize("name", GRIDS)
def test_long_segments(name):
    ny, nz, dt, emf = GRIDS[name]
    p = params(ny, nz)
    assert takes_long(p, 0.75) and takes_long(p, 2.0) == emf
    s = shifts(p, dt)
    assert 0 < s.max() < ny and (ny < 41 or s.max() > 15)
    u0 = fargo_state_for(p, seed=ny)
    fargo_pair(p, u0, dt)
    want, got = updated(p, u0, dt), updated(params(ny, nz, "fp32"), u0, dt)
    for v in range(8):
        assert np.abs(got[..., v] - want[..., v]).max() <= 1e-5 * np.abs(want[..., v]).max(), v


def checked():
    assert dg.load_library().dg_debug_oob_count() == 0, "not the checked build"
    for ny, nz, dt, _ in GRIDS.values():
        u0 = fargo_state_for(params(ny, nz), seed=ny)
        for precision in ("fp64", "fp32"):
            assert np.isfinite(updated(params(ny, nz, precision), u0, dt)[..., :8]).all()
    print("OOB", dg.load_library().dg_debug_oob_count())


def test_checked_build_has_no_out_of_range_access():
    from dumses_hybrid_b200 import build
    child = "import sys; sys.path[:0] = sys.argv[1:3]; import test_fargo_segments_gpu as t; t.checked()"
    res = subprocess.run([sys.executable, "-c", child, str(HERE.parent), str(HERE)], capture_output=True, text=True,
                         timeout=600, env=dict(os.environ, DG_LIBRARY=str(build.LIB_CHK)))
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-4000:]
    assert "OOB 0" in res.stdout, res.stdout[-2000:]
