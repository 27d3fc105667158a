"""The straight-line FP64 solves (csrc/round64.cuh) against the oracle, bit for bit, where their
operands leave the range they are good for and the solves go back to the IEEE operators: quotients
and squares beyond 2^+-200, numerators that are zero or far below 2^-700, and both kinds of cell side
by side; fans that lie wholly on one side of an interface; and operands a few ulps from 1, whose quotients
and roots lie next to rounding ties."""
import numpy as np
import pytest

from dumses_hybrid_b200 import Context, Params, condinit
from _oracle import Oracle
from test_parity_gpu import compare_states

pytestmark = pytest.mark.gpu


def base(iso):
    kw = dict(iso=1, ciso=1.0) if iso else {}
    p = Params(ndim=3, nx=17, ny=12, nz=9, xmin=0, xmax=1, ymin=0, ymax=1, zmin=0, zmax=1, courant=0.4, **kw)
    u = condinit(p, "orszag_tang")
    rng = np.random.default_rng(3)
    u[..., 3] += 0.1 * u[..., 0] * np.sin(2 * np.pi * rng.random(u.shape[2]))[None, None, :]
    return p, u


def set_energy(u, pressure):
    kin = 0.5 * (u[..., 1] ** 2 + u[..., 2] ** 2 + u[..., 3] ** 2) / u[..., 0]
    mag = sum(0.5 * (0.5 * (u[..., 5 + c] + u[..., 8 + c])) ** 2 for c in range(3))
    u[..., 4] = pressure / (5.0 / 3.0 - 1.0) + kin + mag


def variant(name, u):
    half = np.zeros(u.shape[:3], bool)
    half[: u.shape[0] // 2] = True
    rng = np.random.default_rng(5)
    if name == "units_large":    # velocities x 2^60: the squared squares pass 2^200
        u[..., 1:4] *= 2.0**60
        u[..., 4] *= 2.0**120
        u[..., 5:] *= 2.0**60
    elif name == "units_small":
        u[..., 1:4] *= 2.0**-60
        u[..., 4] *= 2.0**-120
        u[..., 5:] *= 2.0**-60
    elif name == "tiny_field":   # quotients of numbers far below 2^-700
        u[..., 5:] *= 1e-250
        set_energy(u, 0.3)
    elif name == "denormal_field":
        u[..., 5:] *= 1e-312
        set_energy(u, 0.3)
    elif name == "zero_half":    # no field and no flow in one half
        u[half, 1:4] = 0.0
        u[half, 5:] = 0.0
        set_energy(u, 0.3)
    elif name == "mixed_cells":  # either kind next to the other
        pick = rng.random(u.shape[:3]) < 0.3
        u[pick, 5:] *= 1e-260
        u[pick, 1:4] *= 1e-130
        set_energy(u, 0.3)
    elif name == "supersonic":   # the whole fan on one side of a face
        u[..., 1] += 30.0 * u[..., 0]
        u[..., 2] -= 30.0 * u[..., 0]
        set_energy(u, 0.3)
    elif name == "near_unity":   # density and pressure of 1 to within rounding: quotients and roots next to ties
        eps = np.ldexp(rng.integers(-3, 4, u.shape[:3]).astype(float), -53)
        u[..., 0] = 1.0 + eps
        u[..., 1], u[..., 2], u[..., 3] = 2.0, 1.0, 0.0
        u[..., 5:] *= 1e-3
        set_energy(u, 1.0)
    elif name == "strong_field":  # Alfven speed far above the sound speed, field along z
        u[..., 7] = u[..., 10] = 40.0
        set_energy(u, 0.3)
    return u


@pytest.mark.parametrize("iso", [False, True])
@pytest.mark.parametrize("name", ["plain", "units_large", "units_small", "tiny_field", "denormal_field", "zero_half",
                                  "mixed_cells", "supersonic", "near_unity", "strong_field"])
def test_solves_outside_the_straight_line_range(name, iso):
    p, u0 = base(iso)
    if iso and name.startswith("units"):
        p.ciso = 2.0**60 if name == "units_large" else 2.0**-60
    u0 = np.asfortranarray(variant(name, u0))
    o = Oracle(p)
    o.set_state(u0)
    o.boundary(0.0, 0.0)
    t = 0.0
    for _ in range(2):
        t, _ = o.step(t)
    with Context(p) as g:
        g.upload(u0)
        g.boundary(0.0, 0.0)
        tg, _ = g.run(2, 0.0)
        ug = g.download()
    assert tg == t
    compare_states(ug, o.uin, p)


@pytest.mark.parametrize("iso", [False, True])
@pytest.mark.parametrize("name", ["units_large", "tiny_field", "mixed_cells", "near_unity"])
def test_2d_solves_outside_the_straight_line_range(name, iso):
    kw = dict(iso=1, ciso=2.0**60 if name == "units_large" else 1.0) if iso else {}
    p = Params(ndim=2, nx=33, ny=18, nz=1, xmin=0, xmax=1, ymin=0, ymax=1, courant=0.4, **kw)
    u0 = np.asfortranarray(variant(name, condinit(p, "field_loop")))
    o = Oracle(p)
    o.set_state(u0)
    o.boundary(0.0, 0.0)
    t = 0.0
    for _ in range(2):
        t, _ = o.step(t)
    with Context(p) as g:
        g.upload(u0)
        g.boundary(0.0, 0.0)
        tg, _ = g.run(2, 0.0)
        ug = g.download()
    assert tg == t
    compare_states(ug, o.uin, p)
