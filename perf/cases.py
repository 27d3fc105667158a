"""The work this package does for its users, as cases that can be timed and checked.

Four kinds of program call the package:

``run``    a simulation whose state stays on the device: a batch of steps (``Context.run``),
           then the state back on the host in the reference layout for a dump.  The next
           batch goes on from there.
``loop``   the reference's own driver loop: the state comes from the host, and every step
           calls ``compute_dt`` (dt is read back), ``godunov``, ``fargo_update``, ``boundary``
           and ``dissipation``; at the end the history sums and the state.
``train``  Adam steps of the flux network on samples kept on the device.
``grad``   one forward and backward pass of the flux network on a batch from the host.

The flows are the package's benchmark and test problems: the isothermal shearing box with a
net vertical field and FARGO ("mri"), the three-dimensional Orszag-Tang vortex ("ot") and the
two-dimensional advected field loop ("loop2d").  :func:`exact` evolves the same initial state
with the same scheme (MUSCL-Hancock, MC slopes, HLLD faces and edges, constrained transport)
written in plain torch in 64 bits.
"""
import functools
import math

import numpy as np
import torch

from dumses_hybrid_b200 import Context, FluxNet, Params

PI = math.pi
R, U, V, W, P, A, B, C = range(8)


def _case(name, kind, flow, nx, ny, nz, steps, precision="fp64", net=False, nu=0.0, eta=0.0, batch=0):
    c = {"kind": kind, "flow": flow, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "precision": precision,
         "net": net, "nu": nu, "eta": eta, "batch": batch}
    return {"name": name, **c} if name else c


def listed():
    return [
        # 2D field loop, 128 x 64: the smallest grid in use, where launches and latency count
        _case("loop2d_128x64_fp64", "run", "loop2d", 128, 64, 1, 60),
        # the reference's driver loop on its regression grid, dt read back at every step
        _case("driver_mri_32x64x32_fp64", "loop", "mri", 32, 64, 32, 12),
        # a small periodic box, as in parameter studies and tests
        _case("ot_64_fp64", "run", "ot", 64, 64, 64, 40),
        # odd extents that fill no tile, FP32
        _case("ot_101x75x53_fp32", "run", "ot", 101, 75, 53, 60, "fp32"),
        # viscosity and resistivity switched on, odd extents, through the driver loop
        _case("driver_mri_diss_90x126x70_fp64", "loop", "mri", 90, 126, 70, 10, nu=1e-4, eta=1e-4),
        # the shearing-box turbulence box (128 x 256 x 128) in both arithmetics
        _case("mri_128x256x128_fp64", "run", "mri", 128, 256, 128, 40),
        _case("mri_128x256x128_fp32", "run", "mri", 128, 256, 128, 60, "fp32"),
        # 256^3: the vortex in FP64, the shearing box in FP32 and with the learned face flux
        _case("ot_256_fp64", "run", "ot", 256, 256, 256, 16),
        _case("mri_256_fp32", "run", "mri", 256, 256, 256, 32, "fp32"),
        _case("mri_256_fp32_net", "run", "mri", 256, 256, 256, 20, "fp32", net=True),
        # training of the flux network at its batch size, and a single gradient
        _case("train_65536", "train", "mri", 48, 48, 48, 40, "fp32", net=True, batch=65536),
        _case("grad_16384", "grad", "mri", 48, 48, 48, 1, "fp32", net=True, batch=16384),
    ]


def draw(rng):
    what = rng.choice(["run", "run", "run", "loop", "net", "loop2d", "train"])

    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if what == "loop2d":
        nx, ny = side(48, 1024), side(24, 512)
        return _case(None, "run", "loop2d", nx, ny, 1, max(8, min(80, 4000000 // (nx * ny))), rng.choice(["fp64", "fp32"]))
    if what == "train":
        return _case(None, "train", "mri", 48, 48, 48, rng.randint(10, 40), "fp32", net=True,
                     batch=128 * side(16, 512))
    nx, ny, nz = side(20, 256), side(20, 256), side(20, 256)
    steps = max(3, min(16, 60000000 // (nx * ny * nz)))
    flow = rng.choice(["mri", "ot"])
    if what == "net":
        return _case(None, "run", "mri", nx, ny, nz, steps, "fp32", net=True)
    if what == "loop":
        nu = rng.choice([0.0, 1e-4])
        return _case(None, "loop", flow, nx, ny, nz, max(3, steps // 2), rng.choice(["fp64", "fp32"]), nu=nu, eta=nu)
    return _case(None, "run", flow, nx, ny, nz, steps, rng.choice(["fp64", "fp32"]))


def work(case):
    if case["kind"] in ("train", "grad"):
        weights = 17 * 64 + 64 * 64 + 64 * 8
        n = case["batch"] * case["steps"]
        return {"bytes": n * (17 + 8) * 4.0, "flops": 6.0 * weights * n}
    cells = case["nx"] * case["ny"] * case["nz"]
    # the 8 conserved variables read and written once a step (64 bits each, or a pair of 32), and
    # the 11 variables of the final state; about 2600 operations a cell and step in 3D
    return {"bytes": 128.0 * cells * case["steps"] + 2 * 88.0 * cells,
            "flops": (2600.0 if case["nz"] > 1 else 1000.0) * cells * case["steps"]}


# ---------------------------------------------------------------------------------------------
# the initial states, on the device in the reference's variable order
# ---------------------------------------------------------------------------------------------
class Box:
    """Extents, spacings and constants of a case's grid; arrays are [k, j, i] with 3 ghost cells."""

    def __init__(self, case):
        self.nx, self.ny, self.nz = case["nx"], case["ny"], case["nz"]
        self.flow, self.two_d = case["flow"], case["flow"] == "loop2d"
        n = (self.nx, self.ny, self.nz)
        if self.flow == "mri":  # the box's shape follows its extents: cubic cells, unit length along y
            h = 1.0 / self.ny
            self.lo, self.hi = [-0.5 * m * h for m in n], [0.5 * m * h for m in n]
        elif self.flow == "ot":
            self.lo, self.hi = [0.0] * 3, [1.0] * 3
        else:
            self.lo, self.hi = [-1.0, -0.5, 0.0], [1.0, 0.5, 1.0]
        self.d = [(b - a) / m for a, b, m in zip(self.lo, self.hi, n)]
        self.iso = self.flow == "mri"
        self.gamma, self.ciso = 5.0 / 3.0, (1.0 if self.iso else 0.0)
        self.omega = 1.0 if self.iso else 0.0
        self.cfl = 0.7 if self.two_d else 0.8
        self.nu, self.eta = case["nu"], case["eta"]
        self.gz = 0 if self.two_d else 3
        self.shape = (self.nz + 2 * self.gz, self.ny + 6, self.nx + 6)

    def centres(self):
        """x, y, z of the cell centres, ghosts included, shaped for broadcasting."""
        out = []
        for a, (n, g) in enumerate(((self.nx, 3), (self.ny, 3), (self.nz, self.gz))):
            i = torch.arange(n + 2 * g, dtype=torch.float64, device="cuda") - g
            s = [1, 1, 1]
            s[2 - a] = -1
            out.append((self.lo[a] + self.d[a] / 2 + i * self.d[a]).reshape(s))
        return out

    def params(self, case):
        p = Params(ndim=2 if self.two_d else 3, iso=int(self.iso), nx=self.nx, ny=self.ny, nz=self.nz, xmin=self.lo[0],
                   xmax=self.hi[0], ymin=self.lo[1], ymax=self.hi[1], zmin=self.lo[2], zmax=self.hi[2],
                   gamma=self.gamma, ciso=self.ciso, omega0=self.omega, courant=self.cfl, slope_type=2,
                   precision=case["precision"], surrogate=bool(case["net"]), nu=self.nu, eta=self.eta)
        if self.iso:
            p.bdtypex, p.fargo = "shearingbox", True
        return p


def initial(box, seed):
    """The eight conserved variables (left-face field) of a case's flow, ghosts not yet filled."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    u = torch.zeros((8,) + box.shape, dtype=torch.float64, device="cuda")
    x, y, z = box.centres()
    one = torch.ones(box.shape, dtype=torch.float64, device="cuda")
    rnd = torch.rand(8, generator=g, device="cuda", dtype=torch.float64)
    if box.flow == "mri":
        u[R] = 1.0
        u[U:P] = 0.1 * (torch.rand((3,) + box.shape, generator=g, device="cuda", dtype=torch.float64) - 0.5)
        u[C] = math.sqrt(2.0 / 1000.0)
    elif box.flow == "ot":
        rho, b0 = 25.0 / (36.0 * PI), 1.0 / math.sqrt(4.0 * PI)
        vx = -torch.sin(2 * PI * y) * one + 0.05 * torch.cos(2 * PI * (z + rnd[0]))
        vy = torch.sin(2 * PI * x) * one + 0.05 * torch.cos(2 * PI * (z + rnd[1]))
        vz = 0.2 * torch.sin(2 * PI * (z + rnd[2])) * one
        u[R], u[U], u[V], u[W] = rho, rho * vx, rho * vy, rho * vz
        u[A], u[B] = -b0 * torch.sin(2 * PI * y) * one, b0 * torch.sin(4 * PI * x) * one
        u[P] = 5.0 / (12.0 * PI) / (box.gamma - 1) + 0.5 * rho * (vx**2 + vy**2 + vz**2) + 0.5 * (u[A]**2 + u[B]**2)
    else:
        cx, cy = 2.0 * float(rnd[0]) - 1.0, float(rnd[1]) - 0.5

        def near(q, c, length):  # distance along a periodic axis
            return torch.remainder(q - c + 0.5 * length, length) - 0.5 * length

        def az(xx, yy):
            return 1e-3 * torch.clamp(0.3 - torch.sqrt(near(xx, cx, 2.0)**2 + near(yy, cy, 1.0)**2), min=0.0)

        dx, dy = box.d[0], box.d[1]
        a0, ax, ay, axy = az(x, y), az(x + dx, y), az(x, y + dy), az(x + dx, y + dy)
        u[R], u[U], u[V] = 1.0, 2.0, 1.0
        u[A], u[B] = (ay - a0) / dy, -(ax - a0) / dx
        bx, by = 0.5 * (ay - a0 + axy - ax) / dy, -0.5 * (ax - a0 + axy - ay) / dx
        u[P] = 1.0 / (box.gamma - 1) + 2.5 + 0.5 * (bx**2 + by**2)
    return u


def reference_layout(u):
    """uin(i, j, k, 1:11) as a [variable, k, j, i] array: the right faces are the next cell's left ones."""
    right = []
    for v, axis in ((A, 2), (B, 1), (C, 0)):
        r = torch.roll(u[v], -1, axis)
        last = [slice(None)] * 3
        last[axis] = -1
        r[tuple(last)] = u[v][tuple(last)]
        right.append(r)
    return torch.cat([u, torch.stack(right)])


# ---------------------------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------------------------
def _host(u):
    """A pinned host array in the reference layout, and its Fortran-ordered numpy view."""
    t = torch.empty(u.shape, dtype=torch.float64, pin_memory=True)
    t.copy_(u)
    return t, t.numpy().T


def prepare(case, seed):
    if case["kind"] in ("train", "grad"):
        x, t = interface_samples(int(seed))
        s = {"case": case, "net": FluxNet(seed=5)}
        if case["kind"] == "grad":
            pick = np.random.default_rng(seed).integers(0, x.shape[0], case["batch"])
            s["x"], s["t"] = np.ascontiguousarray(x[pick]), np.ascontiguousarray(t[pick])
        else:
            s["net"].set_samples(x, t)
            s["net"].fit_scaling()
        s["net"].set_params(first_params(int(seed)))
        return s
    box = Box(case)
    s = {"case": case, "ctx": Context(box.params(case)), "t": 0.0}
    s["uin"], s["view"] = _host(reference_layout(initial(box, seed)))
    s["ctx"].upload(s["view"])
    s["ctx"].boundary(0.0, 0.0)
    if case["kind"] == "loop":  # the driver keeps its own copy of the initial state
        s["ctx"].download_into(s["view"])
        s["u0"], s["v0"] = _host(s["uin"])
    if case["net"]:
        s["net"] = trained_net()
        s["ctx"].attach_surrogate(s["net"])
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "train":
        loss = s["net"].train(case["steps"], batch=case["batch"], lr=1e-3)
        return {"params": s["net"].params(), "loss": np.float32(loss)}
    if case["kind"] == "grad":
        loss, grad = s["net"].gradients(s["x"], s["t"])
        return {"loss": np.float32(loss), "grad": grad}
    ctx = s["ctx"]
    if case["kind"] == "run":
        s["t"], _ = ctx.run(case["steps"], s["t"])
        ctx.download_into(s["view"])
        return s["uin"]
    ctx.upload(s["v0"])
    time = 0.0
    for _ in range(case["steps"]):
        dt = ctx.compute_dt()
        ctx.godunov(dt, time)
        if ctx.params.fargo:
            ctx.fargo_update(dt)
        ctx.boundary(time, dt)
        if case["nu"] > 0.0 or case["eta"] > 0.0:
            ctx.dissipation(time, dt)
        time += dt
    sums = ctx.history()
    ctx.download_into(s["view"])
    return {"history": sums, "uin": s["uin"]}


# ---------------------------------------------------------------------------------------------
# the scheme in plain torch, 64 bits
# ---------------------------------------------------------------------------------------------
def sh(a, axis, n):
    """a at index + n along axis (0 = x, 1 = y, 2 = z)."""
    return torch.roll(a, -n, a.dim() - 1 - axis)


def mc(m, c, p):
    dl, dr = 2.0 * (c - m), 2.0 * (p - c)
    cen = 0.25 * (dl + dr)
    lim = torch.where(dl * dr <= 0, torch.zeros_like(dl), torch.minimum(dl.abs(), dr.abs()))
    return torch.copysign(torch.minimum(lim, cen.abs()), cen)


def half_slope(a, axis):
    return 0.5 * mc(sh(a, axis, -1), a, sh(a, axis, 1))


SMALLR = 1e-10


def fast2(gamma, p, r, bn, b2):
    c2 = gamma * p / r
    d2 = 0.5 * (c2 + b2 / r)
    return d2 + torch.sqrt(torch.clamp(d2 * d2 - c2 * bn * bn / r, min=0.0))


def hlld(L, Rt, bn, gamma):
    """Fluxes (rho, E, u, v, w without the total pressure) and the star total pressure; states r, p, u, v, w, b, c."""
    S = []
    for r, p, u, v, w, b, c in (L, Rt):
        b2 = bn * bn + b * b + c * c
        e = p / (gamma - 1) + 0.5 * r * (u * u + v * v + w * w) + 0.5 * b2
        S.append((r, p, u, v, w, b, c, e, p + 0.5 * b2, u * bn + v * b + w * c))
    (rl, pl, ul, vl, wl, bl, cl, el, tl, xl), (rr, pr, ur, vr, wr, br, cr, er, tr, xr) = S
    cf = torch.sqrt(torch.maximum(fast2(gamma, pl, rl, bn, bn * bn + bl * bl + cl * cl),
                                  fast2(gamma, pr, rr, bn, bn * bn + br * br + cr * cr)))
    sl, sr = torch.minimum(ul, ur) - cf, torch.maximum(ul, ur) + cf
    kl, kr = rl * (ul - sl), rr * (sr - ur)
    us = (kr * ur + kl * ul + (tl - tr)) / (kr + kl)
    ts = (kr * tl + kl * tr + kl * kr * (ul - ur)) / (kr + kl)
    star = []
    for (r, p, u, v, w, b, c, e, t, x), s in zip(S, (sl, sr)):
        rs = r * (s - u) / (s - us)
        q = r * (s - u) * (s - us) - bn * bn
        f = r * (s - u) * (s - u) - bn * bn
        z = q == 0
        q = torch.where(z, torch.ones_like(q), q)
        g = torch.where(z, torch.zeros_like(q), bn * (us - u) / q)
        h = torch.where(z, torch.ones_like(q), f / q)
        vs, ws, bs, cs = v - b * g, w - c * g, b * h, c * h
        xs = us * bn + vs * bs + ws * cs
        es = ((s - u) * e - t * u + ts * us + bn * (x - xs)) / (s - us)
        star.append((rs, vs, ws, bs, cs, xs, es, torch.sqrt(rs)))
    (rsl, vsl, wsl, bsl, csl, xsl, esl, ql), (rsr, vsr, wsr, bsr, csr, xsr, esr, qr) = star
    sg = torch.copysign(torch.ones_like(bn), bn)
    al, ar = us - bn.abs() / ql, us + bn.abs() / qr
    v2 = (ql * vsl + qr * vsr + sg * (bsr - bsl)) / (ql + qr)
    w2 = (ql * wsl + qr * wsr + sg * (csr - csl)) / (ql + qr)
    b2 = (ql * bsr + qr * bsl + sg * ql * qr * (vsr - vsl)) / (ql + qr)
    c2 = (ql * csr + qr * csl + sg * ql * qr * (wsr - wsl)) / (ql + qr)
    x2 = us * bn + v2 * b2 + w2 * c2
    e2l, e2r = esl - sg * ql * (xsl - x2), esr + sg * qr * (xsr - x2)
    zones = [(sl, (rl, ul, vl, wl, bl, cl, tl, el, xl)), (al, (rsl, us, vsl, wsl, bsl, csl, ts, esl, xsl)),
             (us, (rsl, us, v2, w2, b2, c2, ts, e2l, x2)), (ar, (rsr, us, v2, w2, b2, c2, ts, e2r, x2)),
             (sr, (rsr, us, vsr, wsr, bsr, csr, ts, esr, xsr))]
    o = (rr, ur, vr, wr, br, cr, tr, er, xr)
    for s, st in reversed(zones):
        o = tuple(torch.where(s > 0, a, b) for a, b in zip(st, o))
    r, u, v, w, b, c, t, e, x = o
    return [r * u, (e + t) * u - bn * x, r * u * u - bn * bn, r * u * v - bn * b, r * u * w - bn * c], t


def hlld_edge(q, gamma):
    """EMF of an edge from its four corner states r, p, u, v, A, B, C (keys LL, LR, RL, RR)."""
    K = ("LL", "LR", "RL", "RR")
    E = {k: q[k][2] * q[k][5] - q[k][3] * q[k][4] for k in K}
    pt, fx, fy = {}, [], []
    for k in K:
        r, p, u, v, a, b, c = q[k]
        b2 = a * a + b * b + c * c
        pt[k] = p + 0.5 * b2
        fx.append(fast2(gamma, p, r, a, b2))
        fy.append(fast2(gamma, p, r, b, b2))

    def ext(f, vals):
        return functools.reduce(f, vals)

    cx, cy = torch.sqrt(ext(torch.maximum, fx)), torch.sqrt(ext(torch.maximum, fy))
    us_, vs_ = [q[k][2] for k in K], [q[k][3] for k in K]
    SX = {"L": ext(torch.minimum, us_) - cx, "R": ext(torch.maximum, us_) + cx}
    SY = {"L": ext(torch.minimum, vs_) - cy, "R": ext(torch.maximum, vs_) + cy}
    kx = {k: q[k][0] * (q[k][2] - SX["L"] if k[0] == "L" else SX["R"] - q[k][2]) for k in K}
    ky = {k: q[k][0] * (q[k][3] - SY["L"] if k[1] == "L" else SY["R"] - q[k][3]) for k in K}
    us = (sum(kx[k] * q[k][2] for k in K) + (pt["LL"] - pt["RL"] + pt["LR"] - pt["RR"])) / sum(kx.values())
    vs = (sum(ky[k] * q[k][3] for k in K) + (pt["LL"] - pt["LR"] + pt["RL"] - pt["RR"])) / sum(ky.values())
    As, Bs, Ex, Ey, Es, ax, ay = {}, {}, {}, {}, {}, {}, {}
    for k in K:
        r, p, u, v, a, b, c = q[k]
        gx, gy = (SX[k[0]] - u) / (SX[k[0]] - us), (SY[k[1]] - v) / (SY[k[1]] - vs)
        Bs[k], As[k] = b * gx, a * gy
        Ex[k], Ey[k], Es[k] = us * Bs[k] - v * a, u * b - vs * As[k], us * Bs[k] - vs * As[k]
        rs = torch.sqrt(r * gx * gy)
        ax[k] = torch.maximum(a.abs() / torch.sqrt(r * gx), As[k].abs() / rs)
        ay[k] = torch.maximum(b.abs() / torch.sqrt(r * gy), Bs[k].abs() / rs)
    low = 1e-10
    sal = torch.clamp(us - torch.clamp(torch.maximum(ax["LL"], ax["LR"]), min=low), max=0.0)
    sar = torch.clamp(us + torch.clamp(torch.maximum(ax["RL"], ax["RR"]), min=low), min=0.0)
    sab = torch.clamp(vs - torch.clamp(torch.maximum(ay["LL"], ay["RL"]), min=low), max=0.0)
    sat = torch.clamp(vs + torch.clamp(torch.maximum(ay["LR"], ay["RR"]), min=low), min=0.0)
    dx, dy = sar - sal, sat - sab

    def along_x(l, r):
        return (sar * Ex[l] - sal * Ex[r] + sar * sal * (q[r][5] - q[l][5])) / dx

    def along_y(b, t):
        return (sat * Ey[b] - sab * Ey[t] - sat * sab * (q[t][4] - q[b][4])) / dy

    at, ab = (sar * As["RR"] - sal * As["LR"]) / dx, (sar * As["RL"] - sal * As["LL"]) / dx
    br, bl = (sat * Bs["RR"] - sab * Bs["RL"]) / dy, (sat * Bs["LR"] - sab * Bs["LL"]) / dy
    mid = ((sal * sab * Es["RR"] - sal * sat * Es["RL"] - sar * sab * Es["LR"] + sar * sat * Es["LL"]) / dx / dy
           - sat * sab / dy * (at - ab) + sar * sal / dx * (br - bl))
    w = torch.where
    left, right, low_, high = SX["L"] > 0, SX["R"] < 0, SY["L"] > 0, SY["R"] < 0
    return w(low_, w(left, E["LL"], w(right, E["RL"], along_x("LL", "RL"))),
             w(high, w(left, E["LR"], w(right, E["RR"], along_x("LR", "RR"))),
               w(left, along_y("LL", "LR"), w(right, along_y("RL", "RR"), mid))))


class Exact:
    """One flow, stepped as the reference's loop body does."""

    def __init__(self, box, seed):
        self.b, self.u, self.t = box, initial(box, seed), 0.0
        nx, ny, nz, gz = box.nx, box.ny, box.nz, box.gz
        self.act = (slice(gz, gz + nz), slice(3, 3 + ny), slice(3, 3 + nx))
        # rows and columns that hold the cells 1..n+1 (the faces of the active cells)
        self.face = (slice(gz, gz + nz + (gz > 0)), slice(3, 4 + ny), slice(3, 4 + nx))
        self.fill(0.0)

    def shear(self, time):
        b = self.b
        dy = math.fmod(1.5 * b.omega * (b.hi[0] - b.lo[0]) * time, b.hi[1] - b.lo[1])
        return math.fmod(dy, b.d[1]), int(dy / b.d[1])

    def rows(self, a, shift):
        """Rows of the active y range, row j reading row j + shift (periodic)."""
        return torch.roll(a[..., 3:3 + self.b.ny, :], -shift, -2)

    def fill(self, time):
        b, u, nx, ny, nz, gz = self.b, self.u, self.b.nx, self.b.ny, self.b.nz, self.b.gz
        if b.iso:
            epsi, jp = self.shear(time)
            outer = u[A, :, :, 3 + nx].clone()
            for lower in (True, False):
                src = u[..., nx:nx + 3] if lower else u[..., 3:6]
                sh_ = -(jp + 1) if lower else jp
                eps = 1.0 - epsi / b.d[1] if lower else epsi / b.d[1]
                lam = 0.5 * eps * (eps - 1.0)
                a0, a1 = self.rows(src, sh_), self.rows(src, sh_ + 1)
                am, a2 = self.rows(src, sh_ - 1), self.rows(src, sh_ + 2)
                s0, s1 = mc(am, a0, a1), mc(a0, a1, a2)
                val = (1 - eps) * a0 + eps * a1 + lam * (s0 - s1 if lower else s1 - s0)
                val[B] = a0[B] + eps * (a1[B] - a0[B])
                u[..., 3:3 + ny, (0 if lower else nx + 3):(3 if lower else nx + 6)] = val
            u[A, :, :, 3 + nx] = outer
        else:
            u[..., :3], u[..., nx + 3:] = u[..., nx:nx + 3].clone(), u[..., 3:6].clone()
        u[..., :3, :], u[..., ny + 3:, :] = u[..., ny:ny + 3, :].clone(), u[..., 3:6, :].clone()
        if gz:
            u[:, :3], u[:, nz + 3:] = u[:, nz:nz + 3].clone(), u[:, 3:6].clone()

    def prim(self):
        b, u = self.b, self.u
        q = torch.empty_like(u)
        q[R] = torch.clamp(u[R], min=SMALLR)
        q[U:P] = u[U:P] / u[R]
        for v, axis in ((A, 0), (B, 1), (C, 2)):
            q[v] = 0.5 * (u[v] + sh(u[v], axis, 1))
        if b.iso:
            q[P] = u[R] * b.ciso**2
        else:
            ek, em = 0.5 * (q[U:P]**2).sum(0), 0.5 * (q[A:]**2).sum(0)
            q[P] = torch.clamp((b.gamma - 1) * q[R] * ((u[P] - em) / u[R] - ek), min=1e-30 / b.gamma)
        return q

    def cfl(self, q):
        b, s = self.b, 0.0
        b2 = (q[A:]**2).sum(0)
        for a in range(2 if b.two_d else 3):
            s = s + (torch.sqrt(fast2(b.gamma, q[P], q[R], q[A + a], b2)) + q[U + a].abs()) / b.d[a]
        return b.cfl / float(s[self.act].max())

    def trace(self, q, dt):
        """Predicted cell state, half slopes by variable and axis, predicted faces and their slopes."""
        b, f = self.b, self.u
        k = [dt / d for d in b.d]
        if b.two_d:
            k[2] = 0.0
        d = {(v, a): half_slope(q[v], a) for v in range(8) for a in range(3) if v != A + a}
        for a in range(3):
            d[A + a, a] = 0.5 * (sh(f[A + a], a, 1) - f[A + a])
        r, vel, p, fld = q[R], q[U:P], q[P], q[A:]
        st = [torch.empty(0)] * 8
        st[R] = sum((-vel[a] * d[R, a] - d[U + a, a] * r) * k[a] for a in range(3))
        for m in range(3):
            s = 0.0
            for a in range(3):
                if a == m:
                    o = [n for n in range(3) if n != m]
                    g = d[P, a] + sum(fld[n] * d[A + n, a] for n in o)
                    s = s + (-vel[a] * d[U + m, a] - g / r) * k[a]
                else:
                    s = s + (-vel[a] * d[U + m, a] + fld[a] * d[A + m, a] / r) * k[a]
            st[U + m] = s
        st[P] = sum((-vel[a] * d[P, a] - d[U + a, a] * b.gamma * p) * k[a] for a in range(3))
        for m in range(3):
            st[A + m] = sum((vel[m] * d[A + a, a] + fld[a] * d[U + m, a] - vel[a] * d[A + m, a] - fld[m] * d[U + a, a])
                            * k[a] for a in range(3) if a != m)
        cell = [q[v] + st[v] for v in range(8)]
        # edge electric fields and the half-step of the faces
        E = []
        for e in range(3):
            m, n = (e + 1) % 3, (e + 2) % 3

            def avg4(x):
                y = x + sh(x, m, -1)
                return 0.25 * (y + sh(y, n, -1))

            fm, fn = 0.5 * (f[A + m] + sh(f[A + m], n, -1)), 0.5 * (f[A + n] + sh(f[A + n], m, -1))
            E.append(avg4(vel[m]) * fn - avg4(vel[n]) * fm)
        face, fs = [], {}
        for a in range(3):
            m, n = (a + 1) % 3, (a + 2) % 3
            face.append(f[A + a] + 0.5 * ((sh(E[n], m, 1) - E[n]) * k[m] - (sh(E[m], n, 1) - E[m]) * k[n]))
            for o in (m, n):
                fs[a, o] = half_slope(f[A + a], o)
        return cell, d, face, fs, E

    def faces(self, tr, axis):
        cell, d, face, _, _ = tr
        t1, t2 = [n for n in range(3) if n != axis]

        def side(sg):
            s = {v: cell[v] + sg * d[v, axis] for v in range(8) if v != A + axis}
            s[R], s[P] = torch.clamp(s[R], min=SMALLR), torch.clamp(s[P], min=1e-30 / self.b.gamma)
            if self.b.iso:
                s[P] = s[R] * self.b.ciso**2
            o = [s[R], s[P], s[U + axis], s[U + t1], s[U + t2], s[A + t1], s[A + t2]]
            return [sh(x, axis, -1) for x in o] if sg > 0 else o

        # the field on a face is the same seen from both of its cells
        f, pt = hlld(side(+1), side(-1), face[axis], self.b.gamma)
        out = {R: f[0], P: f[1], U + axis: f[2], U + t1: f[3], U + t2: f[4]}
        return out, pt

    def edge(self, tr, e):
        cell, d, face, fs, _ = tr
        m, n = (e + 1) % 3, (e + 2) % 3

        def corner(sm, sn):
            s = {v: cell[v] + sm * d[v, m] + sn * d[v, n] for v in (R, P, U + m, U + n, A + e)}
            s[R], s[P] = torch.clamp(s[R], min=SMALLR), torch.clamp(s[P], min=1e-30 / self.b.gamma)
            if self.b.iso:
                s[P] = s[R] * self.b.ciso**2
            fm = face[m] + sn * fs[m, n]
            fn = face[n] + sm * fs[n, m]
            if sm > 0:
                fm = sh(face[m], m, 1) + sn * sh(fs[m, n], m, 1)
            if sn > 0:
                fn = sh(face[n], n, 1) + sm * sh(fs[n, m], n, 1)
            o = [s[R], s[P], s[U + m], s[U + n], fm, fn, s[A + e]]
            for ax, sg in ((m, sm), (n, sn)):
                if sg > 0:
                    o = [sh(x, ax, -1) for x in o]
            return o

        q = {"LL": corner(1, 1), "RL": corner(-1, 1), "LR": corner(1, -1), "RR": corner(-1, -1)}
        al, ah = 0.5 * (q["LL"][4] + q["RL"][4]), 0.5 * (q["LR"][4] + q["RR"][4])
        bl, bh = 0.5 * (q["LL"][5] + q["LR"][5]), 0.5 * (q["RL"][5] + q["RR"][5])
        for k in q:
            q[k][4], q[k][5] = (al if k[1] == "L" else ah), (bl if k[0] == "L" else bh)
        return hlld_edge(q, self.b.gamma)

    def shear_average(self, a, time):
        """The boundary average of a face quantity between the inner and outer x faces (shearing box)."""
        b = self.b
        epsi, jp = self.shear(time)
        e = epsi / b.d[1]
        lo, hi = a[..., 3].clone(), a[..., 3 + b.nx].clone()

        def row(x, s):
            return torch.roll(x[..., 3:3 + b.ny], -s, -1)

        e0 = 1.0 - e
        lo_new = 0.5 * (row(lo, 0) + (1 - e0) * row(hi, -jp - 1) + e0 * row(hi, -jp))
        hi_new = 0.5 * (row(hi, 0) + (1 - e) * row(lo, jp) + e * row(lo, jp + 1))
        a[..., 3:3 + b.ny, 3], a[..., 3:3 + b.ny, 3 + b.nx] = lo_new, hi_new

    def transport(self, E):
        """Face fields from edge EMFs (already times dt), the edges of the active cells' faces."""
        b, u = self.b, self.u
        for a in range(3):
            m, n = (a + 1) % 3, (a + 2) % 3
            inc = (sh(E[n], m, 1) - E[n]) / b.d[m] - (sh(E[m], n, 1) - E[m]) / b.d[n]
            at = list(self.act)
            at[2 - a] = self.face[2 - a]
            u[A + a][tuple(at)] += inc[tuple(at)]

    def godunov(self, q, dt):
        b, u, act = self.b, self.u, self.act
        if b.omega > 0:
            du, dv = 2 * b.omega * q[V], -0.5 * b.omega * q[U]
            q[U], q[V] = q[U] + du * dt * 0.5, q[V] + dv * dt * 0.5
        tr = self.trace(q, dt)
        dims = range(2 if b.two_d else 3)
        d = {v: 0.0 for v in range(5)}
        lam = 0.25 * (b.omega * dt)**2
        for a in dims:
            f, pt = self.faces(tr, a)
            if b.iso and a == 0:
                self.shear_average(f[R], self.t + 0.5 * dt)
            for v in range(5):
                d[v] = d[v] + ((f[v] - sh(f[v], a, 1)) * dt / b.d[a])[act]
            d[U + a] = d[U + a] + ((pt - sh(pt, a, 1)) * dt / b.d[a])[act]
        none = torch.zeros_like(q[R])
        E = [none if b.two_d and e < 2 else self.edge(tr, e) * dt for e in range(3)]
        if b.iso:
            self.shear_average(E[1], self.t + 0.5 * dt)
        new = [u[v][act] + d[v] for v in range(5)]
        if b.omega > 0:
            mx, my = u[U][act], u[V][act]
            new[U] = (mx * (1 - lam) + 2 * b.omega * dt * my + d[U] + b.omega * dt * d[V]) / (1 + lam)
            new[V] = (my * (1 - lam) - 0.5 * b.omega * dt * mx + d[V] - 0.25 * b.omega * dt * d[U]) / (1 + lam)
        for v in range(5):
            u[v][act] = new[v]
        self.transport(E)

    def fargo(self, dt):
        b, u, ny = self.b, self.u, self.b.ny
        x = b.centres()[0].reshape(-1)
        dy = b.d[1]
        j = torch.arange(ny, device="cuda").reshape(-1, 1)

        def columns(xs):
            v = -1.5 * b.omega * xs
            n = torch.floor((v * dt).abs() / dy).long()
            return v > 0, n, torch.fmod((v * dt).abs(), dy) / dy

        def at(a, idx):  # a[k, j, i] at the row idx[j, i] of each column
            return torch.gather(a, 1, torch.remainder(idx, ny).expand(a.shape[0], -1, -1))

        old = u.clone()
        for half, v, sign in ((0.0, C, 1.0), (0.5 * b.d[0], A, -1.0)):
            up, n, eps = columns(x - half)
            f = old[v][:, 3:3 + ny]
            js = torch.where(up, j - n - 1, j + n)
            w0, w1, w2 = at(f, js - 1), at(f, js), at(f, js + 1)
            frac = eps * w1 + torch.where(up, 0.5 * eps * (1 - eps), 0.5 * eps * (eps - 1)) * mc(w0, w1, w2)
            s = torch.zeros_like(f)
            for m in range(int(n.max())):
                s = s + torch.where(m < n, at(f, torch.where(up, j - 1 - m, j + m)), torch.zeros_like(f))
            out = sign * torch.where(up, s + frac, -s - frac) * dy
            full = torch.zeros_like(old[v])
            full[:, 3:3 + ny] = out
            full[:, 3 + ny] = out[:, 0]
            if v == C:
                ex = full
                ex[3 + b.nz] = ex[3]
            else:
                ez = full
        up, n, eps = columns(x)
        js = torch.where(up, j - n - 1, j + n)
        for v in range(5):
            f = old[v][:, 3:3 + ny]
            a0, a1 = at(f, js), at(f, js + 1)
            s0, s1 = mc(at(f, js - 1), a0, a1), mc(a0, a1, at(f, js + 2))
            h = 0.5 - eps
            val = torch.where(up, a0 * eps + a1 * (1 - eps), a0 * (1 - eps) + a1 * eps)
            val = val + 0.5 * s0 * (0.25 - h * h) + 0.5 * s1 * (h * h - 0.25)
            u[v][self.act] = val[self.act[0], :, self.act[2]]
        self.transport([ex, torch.zeros_like(ex), ez])

    def dissipation(self, time, dt):
        b, u, act = self.b, self.u, self.act

        def diff(x, axis):
            return (x - sh(x, axis, -1)) / b.d[axis]

        if b.eta > 0:
            J = [diff(u[A + (e + 2) % 3], (e + 1) % 3) - diff(u[A + (e + 1) % 3], (e + 2) % 3) for e in range(3)]
            self.transport([-b.eta * x * dt for x in J])
        if b.nu > 0:
            vel = [u[U + m] / u[R] for m in range(3)]
            inc = [0.0] * 4
            for a in range(3):
                rho = 0.5 * (u[R] + sh(u[R], a, -1))
                g = {}
                for m in range(3):
                    if a == 0:  # the reference divides the left momentum by the right cell's density here
                        g[m, a] = (vel[m] - sh(u[U + m], 0, -1) / u[R]) / b.d[0]
                    else:
                        g[m, a] = diff(vel[m], a)
                    for c in range(3):
                        if c != a:
                            y = vel[m] + sh(vel[m], a, -1)
                            g[m, c] = 0.25 * (sh(y, c, 1) - sh(y, c, -1)) / b.d[c]
                o = [c for c in range(3) if c != a]
                tau = {a: -0.66666666666666667 * b.nu * rho * (2 * g[a, a] - g[o[0], o[0]] - g[o[1], o[1]])}
                for c in o:
                    tau[c] = -b.nu * rho * (g[a, c] + g[c, a])
                fl = [tau[m] * dt / b.d[a] for m in range(3)]
                if b.iso:
                    fl.append(torch.zeros_like(rho))
                else:
                    fl.append(sum(0.5 * (vel[m] + sh(vel[m], a, -1)) * tau[m] for m in range(3)) * dt / b.d[a])
                for m in range(4):
                    inc[m] = inc[m] + (fl[m] - sh(fl[m], a, 1))
            for m in range(4):
                u[U + m][act] += inc[m][act]
        self.fill(time + dt)

    def step(self):
        q = self.prim()
        dt = self.cfl(q)
        self.godunov(q, dt)
        if self.b.iso:
            self.fargo(dt)
        self.fill(self.t + dt)
        if self.b.nu > 0 or self.b.eta > 0:
            self.dissipation(self.t, dt)
        self.t += dt

    def history(self):
        """The shearing box's sums: mass, Maxwell and Reynolds stresses, magnetic pressure, mean field, div B."""
        b, u, act = self.b, self.u, self.act
        vol = b.d[0] * b.d[1] * b.d[2] / ((b.hi[0] - b.lo[0]) * (b.hi[1] - b.lo[1]) * (b.hi[2] - b.lo[2]))
        r = u[R][act]
        cen = [(0.5 * (u[v] + sh(u[v], a, 1)))[act] for v, a in ((A, 0), (B, 1), (C, 2))]
        vx, vy = (u[U] / u[R])[act], (u[V] / u[R])[act]
        dv = [v - v.mean((0, 1), keepdim=True) for v in (vx, vy)]
        maxwell, reynolds = -(cen[0] * cen[1]).sum() * vol, (r * dv[0] * dv[1]).sum() * vol
        magp = 0.5 * sum((c * c).sum() for c in cen) * vol
        sums = [r.sum() * vol, maxwell, reynolds, maxwell + reynolds, magp] + [u[v][act].sum() * vol for v in (A, B, C)]
        return torch.tensor([float(x) for x in sums] + [0.0], dtype=torch.float64)


def exact(case, seed):
    if case["kind"] == "train":
        return None
    if case["kind"] == "grad":
        return exact_gradient(case, seed)
    e = Exact(Box(case), seed)
    for _ in range(case["steps"]):
        e.step()
    u = reference_layout(e.u)
    return u if case["kind"] == "run" else {"history": e.history(), "uin": u}


# ---------------------------------------------------------------------------------------------
# the flux network: samples, first parameters, a trained network
# ---------------------------------------------------------------------------------------------
SHAPES = [(17, 64), (64, 64), (64, 8)]
NET_BOX = _case(None, "run", "mri", 48, 48, 48, 0, "fp32")


def interface_samples(seed):
    """Scaled inputs and HLLD-minus-LLF targets of the interfaces of a 48^3 shearing box after a few steps."""
    e = Exact(Box(NET_BOX), seed)
    xs, ts = [], []
    for n in range(9):
        if n in (4, 8):
            q = e.prim()
            dt = e.cfl(q)
            tr = e.trace(q, dt)
            for axis in range(3):
                x, t = _features(e, tr, axis)
                xs.append(x)
                ts.append(t)
        e.step()
    return torch.cat(xs).float().cpu().numpy(), torch.cat(ts).float().cpu().numpy()


def _features(e, tr, axis):
    cell, d, face, _, _ = tr
    g, bn = e.b.gamma, face[axis]
    t1, t2 = [n for n in range(3) if n != axis]

    def side(sg):
        s = {v: cell[v] + sg * d[v, axis] for v in range(8) if v != A + axis}
        o = [s[R], s[R] * e.b.ciso**2, s[U + axis], s[U + t1], s[U + t2], s[A + t1], s[A + t2]]
        return [sh(x, axis, -1) for x in o] if sg > 0 else o

    L, Rt = side(+1), side(-1)
    f, pt = hlld(L, Rt, bn, g)
    (rl, pl, ul, vl, wl, bl, cl), (rr, pr, ur, vr, wr, br, cr) = L, Rt
    cons, flux, tot, vel = [], [], [], []
    for r, p, u, v, w, b, c in (L, Rt):
        b2 = bn * bn + b * b + c * c
        en = p / (g - 1) + 0.5 * r * (u * u + v * v + w * w) + 0.5 * b2
        t = p + 0.5 * b2
        cons.append([r, en, r * u, r * v, b, r * w, c])
        flux.append([r * u, (en + t) * u - bn * (u * bn + v * b + w * c), r * u * u + t - bn * bn, r * u * v - bn * b,
                     b * u - bn * v, r * u * w - bn * c, c * u - bn * w])
        tot.append(t)
        vel.append(torch.sqrt(fast2(g, p, r, bn, b2)) + u.abs())
    vmax = torch.maximum(*vel)
    llf = [0.5 * (a + b) - 0.5 * vmax * (y - x) for a, b, x, y in zip(*flux, *cons)]
    # HLLD's induction fluxes follow from the same wave fan
    bt, ct = _induction(L, Rt, bn, g)
    h = [f[0], f[1], f[2] + pt, f[3], bt, f[4], ct, pt]
    base = llf + [0.5 * (tot[0] + tot[1])]
    rho0 = 0.5 * (rl + rr)
    a0 = torch.sqrt(torch.maximum((g * pl + bn**2 + bl**2 + cl**2) / rl, (g * pr + bn**2 + br**2 + cr**2) / rr))
    b0 = torch.sqrt(rho0) * a0
    units = [rho0, a0, a0, a0, rho0 * a0 * a0, b0, b0]
    ls = [x / y for x, y in zip([rl, ul, vl, wl, pl, bl, cl], units)]
    rs = [x / y for x, y in zip([rr, ur, vr, wr, pr, br, cr], units)]
    dj = [y - x for x, y in zip(ls, rs)]
    jump = torch.sqrt(sum(x * x for x in dj))
    mean = [0.5 * (x + y) for x, y in zip(ls, rs)]
    ind = mean[1:5] + [bn / b0] + mean[5:] + [x / jump for x in dj] + [jump, 0.1 * torch.log(jump),
                                                                       torch.full_like(jump, float(np.float32(g) - np.float32(1)))]
    m = rho0 * a0
    scale = [m, m * a0 * a0, m * a0, m * a0, b0 * a0, m * a0, b0 * a0, m * a0]
    tgt = [(x - y) / (s * jump) for x, y, s in zip(h, base, scale)]
    act = e.act
    return (torch.stack([x[act].reshape(-1) for x in ind], 1), torch.stack([x[act].reshape(-1) for x in tgt], 1))


def _induction(L, Rt, bn, g):
    """HLLD's transverse induction fluxes: the fluxes of the state the fan has at x = 0."""
    # momentum flux and mass flux give the sampled transverse velocity and field only together with
    # the star states, so the fan is sampled again with the passive pair (v, b) and (w, c)
    out = []
    for iv, ib in ((3, 5), (4, 6)):
        r_, S = [], []
        for s in (L, Rt):
            b2 = bn * bn + s[5]**2 + s[6]**2
            S.append((s[0], s[2], s[iv], s[ib], s[1] + 0.5 * b2, fast2(g, s[1], s[0], bn, b2)))
        (rl, ul, vl, bl, tl, fl), (rr, ur, vr, br, tr_, fr) = S
        cf = torch.sqrt(torch.maximum(fl, fr))
        sl, sr = torch.minimum(ul, ur) - cf, torch.maximum(ul, ur) + cf
        kl, kr = rl * (ul - sl), rr * (sr - ur)
        us = (kr * ur + kl * ul + (tl - tr_)) / (kr + kl)
        st = []
        for (r, u, v, b, t, f), s in zip(S, (sl, sr)):
            q = r * (s - u) * (s - us) - bn * bn
            z = q == 0
            q = torch.where(z, torch.ones_like(q), q)
            vs = torch.where(z, v, v - bn * b * (us - u) / q)
            bs = torch.where(z, b, b * (r * (s - u)**2 - bn * bn) / q)
            st.append((vs, bs, torch.sqrt(r * (s - u) / (s - us))))
        (vsl, bsl, ql), (vsr, bsr, qr) = st
        sg = torch.copysign(torch.ones_like(bn), bn)
        v2 = (ql * vsl + qr * vsr + sg * (bsr - bsl)) / (ql + qr)
        b2 = (ql * bsr + qr * bsl + sg * ql * qr * (vsr - vsl)) / (ql + qr)
        o = (ur, vr, br)
        for s, x in ((sr, (us, vsr, bsr)), (us + bn.abs() / qr, (us, v2, b2)), (us, (us, v2, b2)),
                     (us - bn.abs() / ql, (us, vsl, bsl)), (sl, (ul, vl, bl))):
            o = tuple(torch.where(s > 0, a, b) for a, b in zip(x, o))
        out.append(o[2] * o[0] - bn * o[1])
    return out


def first_params(seed):
    """Scaled normal weights and zero biases in the package's parameter order."""
    r = np.random.default_rng(seed)
    return np.concatenate([np.concatenate([(r.standard_normal((k, n)) / math.sqrt(k)).astype(np.float32).reshape(-1),
                                           np.zeros(n, np.float32)]) for k, n in SHAPES])


def _unpack(p):
    out, o = [], 0
    for k, n in SHAPES:
        out.append([p[o:o + k * n].reshape(k, n), p[o + k * n:o + k * n + n]])
        o += k * n + n
    return out


def _smelu(z):
    h = torch.clamp(z, -1.0, 1.0) * 0.5 + 0.5
    return torch.maximum(z, h * h)


def _network(layers, x):
    for n, (w, b) in enumerate(layers):
        x = x @ w + b
        if n + 1 < len(layers):
            x = _smelu(x)
    return x


def exact_gradient(case, seed):
    x, t = interface_samples(int(seed))
    pick = np.random.default_rng(seed).integers(0, x.shape[0], case["batch"])
    x = torch.from_numpy(x[pick]).double().cuda()
    t = torch.from_numpy(t[pick]).double().cuda()
    p = torch.from_numpy(first_params(int(seed))).double().cuda().requires_grad_()
    loss = ((_network(_unpack(p), x) - t)**2).mean()
    loss.backward()
    return {"loss": loss.detach(), "grad": p.grad}


@functools.lru_cache(maxsize=None)
def _trained():
    """Samples and parameters of a network fitted to the interfaces of one shearing box (plain torch)."""
    xs, ts = interface_samples(11)
    x, t = torch.from_numpy(xs).cuda(), torch.from_numpy(ts).cuda()
    mu, sd = x.mean(0), x.std(0).clamp(min=1e-6)
    rms = t.square().mean(0).sqrt()
    x, t = (x - mu) / sd, t / rms
    p = torch.from_numpy(first_params(3)).cuda().requires_grad_()
    opt = torch.optim.Adam([p], lr=2e-3)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    steps = 1500
    for n in range(steps):
        for q in opt.param_groups:
            q["lr"] = 2e-3 * (1.0 - n / steps) + 2e-5
        pick = torch.randint(0, x.shape[0], (16384,), generator=g, device="cuda")
        opt.zero_grad()
        ((_network(_unpack(p), x[pick]) - t[pick])**2).mean().backward()
        opt.step()
    return xs, ts, p.detach().cpu().numpy()


def trained_net():
    """A network as a program loads it: parameters, scaling and envelope."""
    xs, ts, p = _trained()
    net = FluxNet(seed=5)
    net.set_samples(xs, ts)
    net.fit_scaling()
    net.fit_envelope(0.0)
    net.set_params(p)
    return net
