"""The work that a program built on this library has it do, as timed cases.

Each case is one pass through the public entry points (``TGChannel``,
``IOChannel``, ``ChannelBatch``) on fields that are resident on the GPU: time
steps of the periodic (TG) section, of the inflow/outflow (IO) section with
its property and viscous options, of the coupled pair and of the batch, the
substep calls a host program makes one by one, and the on-device statistics.
A pass ends with the fields read back into the program's own device arrays,
as a program that post-processes or writes them does.

Fields have the shape (nz, ny + 2, nx): one wall ghost row on either side,
and in the coupled section one ghost column at either x end.
"""
import math

import numpy as np
import torch

import chapsim1ww_b200 as cs
from chapsim1ww_b200 import ChannelBatch, IOChannel, PropertyEngine, TGChannel, synthetic_table
from chapsim1ww_b200.batch import batch64_configs

DEV = "cuda:0"
LX_TG, LX_IO, LZ = 4 * math.pi, 8 * math.pi, 4 * math.pi / 3
PRT = 0.71
TG_FIELDS = ("u", "v", "w", "p")
IO_FIELDS = ("gx", "gy", "gz", "p", "rhoh", "t")
STAT_FIELDS = ("u", "v", "w", "p", "gx", "gy", "gz", "h", "t", "rho", "mu", "k")


# ------------------------------------------------------------------ the cases
def listed():
    tg = dict(kind="tg", mixed=False, calls=False, steps=1)
    io = dict(kind="io", thermal=True, learned=False, visc=0, isothermal=0, gravdir=0, calls=False, steps=1)
    return [
        # the smallest channel, advanced by a host program that calls the
        # substep routine itself (NS = 1, 2, 3): launch cost and latency
        dict(tg, name="tg_calls_32x24x16", nx=32, ny=24, nz=16, calls=True),
        # the 64^3 channel that is advanced many steps at a time (one graph
        # replay a step)
        dict(tg, name="tg_64x64x64_10steps", nx=64, ny=64, nz=64, steps=10),
        # the production TG channel
        dict(tg, name="tg_256x192x256", nx=256, ny=192, nz=256),
        # lengths with factors 3, 5, 7 and 11, an odd row count, partial tiles
        dict(tg, name="tg_210x99x154", nx=210, ny=99, nz=154),
        # the mixed FP32 / FP64 form of the TG channel
        dict(tg, name="tg_mixed_192x128x160", nx=192, ny=128, nz=160, mixed=True),
        # a small ragged heated IO channel with one iso-thermal wall and
        # buoyancy, its energy and momentum substeps called one by one
        dict(io, name="io_calls_100x49x60", nx=100, ny=49, nz=60, isothermal=1, gravdir=1, calls=True),
        # the heated variable-property channel with the table splines
        dict(io, name="io_384x192x192", nx=384, ny=192, nz=192),
        # the same channel with the semi-implicit viscous scheme
        dict(io, name="io_si_384x192x192", nx=384, ny=192, nz=192, visc=1),
        # the large heated channel with the learned property model (half the
        # span of the 1024 x 384 x 512 domain, so that several states fit)
        dict(io, name="io_learned_1024x384x256", nx=1024, ny=384, nz=256, learned=True),
        # the TG channel feeding the inlet of the IO section: convective
        # outlet, constant-property passive heat
        dict(kind="coupled", name="coupled_256_512x192x256", tgx=256, nx=512, ny=192, nz=256, steps=1),
        # 64 independent channels of uneven sizes, one launch a step
        dict(kind="batch", name="batch_64channels", n=64, sizes=3, steps=1),
        # one sample of the xz and time averages of a heated IO channel
        dict(kind="stats", name="stats_io_384x192x192", nx=384, ny=192, nz=192),
    ]


def _smooth(n, radices=(2, 3, 5, 7, 11)):
    for r in radices:
        while n % r == 0:
            n //= r
    return n == 1


def draw(rng):
    def size(lo, hi):
        """An even length with prime factors up to 11, log-uniform in [lo, hi]."""
        n = 2 * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2))
        while not _smooth(n):
            n += 2
        return n

    def box(cells, xmax=512, ymax=192, zmax=256):
        while True:
            nx, nz = size(24, xmax), size(16, zmax)
            ny = int(round(math.exp(rng.uniform(math.log(20), math.log(ymax)))))
            if nx * ny * nz <= cells:
                return dict(nx=nx, ny=ny, nz=nz)

    kind = rng.choice(["tg", "tg", "tg_mixed", "tg_calls", "io", "io", "io_learned", "io_si", "io_calls", "coupled",
                       "batch", "stats"])
    if kind.startswith("tg"):
        b = box(64 ** 3 if kind == "tg_calls" else 13000000, 384)
        return dict(kind="tg", mixed=kind == "tg_mixed", calls=kind == "tg_calls",
                    steps=10 if b["nx"] * b["ny"] * b["nz"] < 400000 and kind != "tg_calls" else 1, **b)
    if kind.startswith("io"):
        b = box({"io": 20000000, "io_learned": 16000000, "io_si": 8000000, "io_calls": 400000}[kind])
        thermal = kind in ("io_learned",) or rng.random() < 0.8
        # buoyancy in earnest goes with the energy equation
        return dict(kind="io", thermal=thermal, learned=kind == "io_learned", visc=1 if kind == "io_si" else 0,
                    isothermal=rng.choice([0, 1, 2, 3]) if thermal else 0, gravdir=rng.choice([0, 1, 2]) if thermal else 0,
                    calls=kind == "io_calls", steps=1, **b)
    if kind == "coupled":
        b = box(10000000)
        return dict(kind="coupled", tgx=size(24, 256), steps=1, **b)
    if kind == "batch":
        return dict(kind="batch", n=rng.randint(4, 32), sizes=rng.randint(4, 1000), steps=1)
    return dict(kind="stats", **box(14000000))


# ------------------------------------------------------------------ the inputs
def _rows(ny, str2=2.0):
    """Cell centres y_j of the tanh-stretched rows."""
    j = torch.arange(ny, dtype=torch.float64, device=DEV)
    return torch.tanh(str2 * ((j + 0.5) / ny - 0.5)) / math.tanh(str2 * 0.5)


def _velocity(nx, ny, nz, seed, sx=None):
    """The laminar profile with plane-mean-free uniform perturbations of
    amplitude 0.1 and zero wall rows, as (3, nz, ny + 2, sx)."""
    sx = sx or nx
    g = torch.Generator(device=DEV).manual_seed(seed)
    q = torch.zeros((3, nz, ny + 2, sx), dtype=torch.float64, device=DEV)
    for c in range(3):
        r = torch.rand((nz, ny, sx), dtype=torch.float64, device=DEV, generator=g).mul_(0.2).sub_(0.1)
        r -= r.mean(dim=(0, 2), keepdim=True)
        q[c, :, 1:ny + 1] = r
    q[0, :, 1:ny + 1] += (1.5 * (1.0 - _rows(ny) ** 2))[None, :, None]
    q[1, :, 1] = 0.0
    return q


def _enthalpy(nx, ny, nz, seed, span, sx=None):
    """A heated profile with perturbations; the wall ghost rows copy the first
    and last rows."""
    sx = sx or nx
    g = torch.Generator(device=DEV).manual_seed(seed + 7919)
    r = torch.rand((nz, ny, sx), dtype=torch.float64, device=DEV, generator=g).mul_(0.1 * span).sub_(0.05 * span)
    h = torch.empty((nz, ny + 2, sx), dtype=torch.float64, device=DEV)
    h[:, 1:ny + 1] = r + (span * _rows(ny) ** 3)[None, :, None]
    h[:, 0], h[:, ny + 1] = h[:, 1], h[:, ny]
    return h


def _put(ch, **fields):
    torch.cuda.synchronize()  # the context copies on its own stream
    for name, a in fields.items():
        ch.set_field_device(name, a.data_ptr())
    ch.sync()


def _take(ch, name):
    a = torch.empty(ch.shape, dtype=torch.float64, device=DEV)
    torch.cuda.synchronize()
    ch.get_field_device(name, a.data_ptr())
    ch.sync()
    return a


def _buffers(ch, names):
    return {n: torch.empty(ch.shape, dtype=torch.float64, device=DEV) for n in names}


def _start_tg(ch, seed):
    q = _velocity(ch.nx, ch.ny, ch.nz, seed)
    _put(ch, u=q[0], v=q[1], w=q[2])
    ch.solverrk3_mom_tg(0)  # the projection of the initial field
    ch.sync()


_MODEL = {}


def _engine():
    """The property model: 65,536 table samples, seed 2, gated at 1e-4."""
    eng = PropertyEngine(*synthetic_table(4096))
    if "params" not in _MODEL:
        eng.train(65536, 2, 20000, 3e-3)
        _MODEL["params"] = eng.get_params()
    eng.set_params(*_MODEL["params"])
    eng.gate(1e-4, 256)
    return eng


def _constant_table():
    h = np.linspace(-1.0, 1.0, 4096)
    one = np.ones_like(h)
    return h, h.copy(), one, one.copy(), one.copy()


def _io_fields(ch, seed, thermal):
    """The seeded state of an x-periodic IO section before its projection."""
    nx, ny, nz = ch.nx, ch.ny, ch.nz
    q = _velocity(nx, ny, nz, seed)
    if not thermal:
        return dict(u=q[0], v=q[1], w=q[2], gx=q[0], gy=q[1], gz=q[2])
    h = _enthalpy(nx, ny, nz, seed, 0.5)
    _put(ch, h=h)
    ch.therm_prop_update(0)
    props = {n: _take(ch, n) for n in ("t", "rho", "mu", "k")}
    for a in props.values():
        a[:, 0], a[:, ny + 1] = a[:, 1], a[:, ny]
    rho = props["rho"]
    g = [(rho + rho.roll(1, 2)) * 0.5 * q[0], q[1].clone(), (rho + rho.roll(1, 0)) * 0.5 * q[2]]
    g[1][:, 2:ny + 1] *= (rho[:, 2:ny + 1] + rho[:, 1:ny]) * 0.5
    for c in (0, 2):
        g[c][:, 0] = 0.0
        g[c][:, ny + 1] = 0.0
    return dict(u=q[0], v=q[1], w=q[2], gx=g[0], gy=g[1], gz=g[2], h=h, rhoh=rho * h, mu0=props["mu"], rho0=rho,
                **props)


def _stat_fields(nx, ny, nz, seed):
    """The fields that the IO statistics read, with properties of the table's form."""
    q = _velocity(nx, ny, nz, seed)
    h = _enthalpy(nx, ny, nz, seed, 0.5)
    t = 0.9 + 0.5 * h
    rho = 1.0 / (1.0 + 2.0 * t)
    mu = rho ** -0.5
    f = dict(u=q[0], v=q[1], w=q[2], p=0.1 * q[0] * q[0] + q[1], gx=rho * q[0], gy=rho * q[1], gz=rho * q[2], h=h, t=t,
             rho=rho, mu=mu, k=mu * (1.0 + 0.1 * h))
    return {n: f[n].contiguous() for n in STAT_FIELDS}


def _io_channel(case):
    iso = case.get("isothermal", 0)
    # wall temperatures inside the table for the iso-thermal walls, unit
    # fluxes for the others
    qw = (0.60 if iso & 1 else 1.0, 1.20 if iso & 2 else 1.0)
    return IOChannel(case["nx"], case["ny"], case["nz"], lx=LX_IO, lz=LZ, thermal=1 if case["thermal"] else 0, prt=PRT,
                     qw=qw, isothermal=iso, gravdir=case["gravdir"], f_a=0.1 if case["gravdir"] else 0.0,
                     table=synthetic_table(4096) if case["thermal"] else None, visc_scheme=case["visc"])


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "tg":
        ch = TGChannel(case["nx"], case["ny"], case["nz"], lx=LX_TG, lz=LZ,
                       precision=cs.MIXED if case["mixed"] else cs.FP64)
        _start_tg(ch, seed)
        s.update(ch=ch, out=_buffers(ch, TG_FIELDS))
    elif kind == "io":
        ch = _io_channel(case)
        if case["learned"]:
            ch.set_props_mode(1, _engine())
        _put(ch, **_io_fields(ch, seed, case["thermal"]))
        if case["thermal"]:
            ch.solverrk3_eng_io(0)
        ch.solverrk3_mom_io(0)
        ch.sync()
        s.update(ch=ch, out=_buffers(ch, IO_FIELDS if case["thermal"] else IO_FIELDS[:4]))
    elif kind == "coupled":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        tg = TGChannel(case["tgx"], ny, nz, lx=LX_TG, lz=LZ)
        _start_tg(tg, seed)
        ch = IOChannel(nx, ny, nz, lx=LX_IO, lz=LZ, thermal=1, prt=PRT, qw=(1.0, 1.0), table=_constant_table(),
                       bcx=(2, 1))
        ch.set_inlet(tg)
        q = _velocity(nx, ny, nz, seed + 1, nx + 2)
        h = _enthalpy(nx, ny, nz, seed, 0.1, nx + 2)
        _put(ch, u=q[0], v=q[1], w=q[2], gx=q[0], gy=q[1], gz=q[2], h=h, t=h, rhoh=h)
        ch.solverrk3_eng_io(0)
        ch.solverrk3_mom_io(0)
        ch.sync()
        s.update(ch=ch, tg=tg, out=_buffers(ch, IO_FIELDS), tg_out=_buffers(tg, TG_FIELDS))
    elif kind == "batch":
        b = ChannelBatch(batch64_configs(case["sizes"], case["n"]))
        for i, ch in enumerate(b.channels):
            _start_tg(ch, seed + i)
        b.autotune()
        s.update(ch=b, out={f: torch.empty(sum(c.n for c in b.channels), dtype=torch.float64, device=DEV)
                            for f in TG_FIELDS})
    else:
        ch = _io_channel(dict(case, thermal=True, gravdir=0, visc=0))
        _put(ch, **_stat_fields(case["nx"], case["ny"], case["nz"], seed))
        s.update(ch=ch)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def _read(ch, out):
    for name, a in out.items():
        ch.get_field_device(name, a.data_ptr())
    return out


def run(s):
    case, ch = s["case"], s["ch"]
    kind = case["kind"]
    if kind == "tg":
        if case["calls"]:
            for ns in (1, 2, 3):
                ch.solverrk3_mom_tg(ns)
        else:
            ch.step(case["steps"])
        return _read(ch, s["out"])
    if kind == "io":
        if case["calls"]:
            for ns in (1, 2, 3):
                if case["thermal"]:
                    ch.solverrk3_eng_io(ns)
                ch.solverrk3_mom_io(ns)
        else:
            ch.step(case["steps"])
        return _read(ch, s["out"])
    if kind == "coupled":
        ch.step_coupled(s["tg"], case["steps"])
        return {"tg": _read(s["tg"], s["tg_out"]), "io": _read(ch, s["out"])}
    if kind == "batch":
        ch.step(case["steps"])
        at = 0
        for c in ch.channels:
            for name, a in s["out"].items():
                c.get_field_device(name, a.data_ptr() + 8 * at)
            at += c.n
        return s["out"]
    ch.pp_mean_zx(accumulate=True)
    return {"xz": ch.stats(0)[0], "xzt": ch.stats(1)[0]}


# ------------------------------------------------------------------ its cost
def work(case):
    """Every substep ends in a pressure solve over the whole domain, so its
    state is read and written once a substep: TG u, v, w, p and the three old
    convection terms; IO G, p, the three old explicit terms and with the
    energy equation rho h, its old term, h, T, rho, mu, k and the old rho and
    mu.  Flops: the stencils, the line solves, the two transforms each way
    and the 1-64-64-5 network."""
    kind = case["kind"]

    def tg(nx, ny, nz):
        return nx * ny * nz * 2 * 7 * 8.0, nx * ny * nz * (330.0 + 5 * (math.log2(nx) + 2 * math.log2(nz)))

    def io(nx, ny, nz, thermal, learned, visc):
        vals = 2 * 7 + (2 * 9 if thermal else 0)
        fl = 420.0 + 5 * (math.log2(nx) + 2 * math.log2(nz)) + (120.0 if thermal else 0) + (250.0 if visc else 0)
        return nx * ny * nz * vals * 8.0, nx * ny * nz * (fl + (2 * 64 * (1 + 64 + 5) if learned else 0))

    if kind == "stats":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": n * 12 * 8.0 + 2 * case["ny"] * 360 * 8.0, "flops": n * 1000.0}
    if kind == "tg":
        parts = [tg(case["nx"], case["ny"], case["nz"])]
    elif kind == "io":
        parts = [io(case["nx"], case["ny"], case["nz"], case["thermal"], case["learned"], case["visc"])]
    elif kind == "coupled":
        parts = [tg(case["tgx"], case["ny"], case["nz"]), io(case["nx"], case["ny"], case["nz"], True, False, 0)]
    else:
        parts = [tg(c["nx"], c["ny"], c["nz"]) for c in batch64_configs(case["sizes"], case["n"])]
    m = 3.0 * case["steps"]
    return {"bytes": m * sum(p[0] for p in parts), "flops": m * sum(p[1] for p in parts)}


# ------------------------------------------------------------------ 64-bit values
class _TG64:
    """SOLVERRK3_MOM_tg in torch: the cyclic x and z factors and the pressure
    by FFT, the y lines by elimination over all lines at once."""
    GAM, ROH = (1.0, 8 / 15, 5 / 12, 3 / 4), (0.0, 0.0, -17 / 60, -5 / 12)

    def __init__(self, nx, ny, nz, ren, dt, lx=LX_TG):
        self.nx, self.ny, self.nz, self.ren, self.dt = nx, ny, nz, ren, dt
        f64 = dict(dtype=torch.float64, device=DEV)
        self.dxi, self.dzi = nx / lx, nz / LZ
        j = torch.arange(ny + 1, **f64)
        nd, cc = torch.tanh(2.0 * (j / ny - 0.5)) / math.tanh(1.0), _rows(ny)
        self.df = 1.0 / (nd[1:] - nd[:-1])                      # 1 / height of row j
        self.dc = torch.empty(ny + 1, **f64)                    # 1 / distance across face j
        self.dc[1:ny] = 2.0 / (nd[2:] - nd[:-2])
        self.dc[0], self.dc[ny] = 2.0 / (nd[1] - nd[0]), 2.0 / (nd[ny] - nd[ny - 1])
        self.ff, self.fb = torch.zeros(ny + 1, **f64), torch.ones(ny + 1, **f64)  # face weights
        self.ff[1:ny] = (nd[1:ny] - cc[:-1]) / (cc[1:] - cc[:-1])
        self.fb[1:ny] = (cc[1:] - nd[1:ny]) / (cc[1:] - cc[:-1])
        self.ff[ny], self.fb[ny] = 1.0, 0.0
        df, dc = self.df, self.dc
        am, ap = df * dc[:-1], df * dc[1:]
        am[0], ap[-1] = 0.0, 0.0
        self.pois = (am, -(am + ap), ap)
        m, p = df * dc[:-1], df * dc[1:]
        c = -(m + p)
        a = 4.0 / (2.0 / dc[1] + 1.0 / df[0])
        m[0], c[0], p[0] = 0.0, -a * (dc[1] + 2.0 * df[0]), a * dc[1]
        a = 4.0 / (2.0 / dc[ny - 1] + 1.0 / df[ny - 1])
        m[-1], c[-1], p[-1] = a * dc[ny - 1], -a * (2.0 * df[-1] + dc[ny - 1]), 0.0
        mv, pv = torch.zeros(ny, **f64), torch.zeros(ny, **f64)
        mv[1:], pv[1:] = df[:-1] * dc[1:ny], df[1:] * dc[1:ny]
        cv = -(mv + pv)
        cv[0] = 1.0
        self.visc = ((m, c, p), (mv, cv, pv), (m, c, p))
        wave = lambda n: 2.0 * (1.0 - torch.cos(2.0 * math.pi * torch.arange(n, **f64) / n))  # noqa: E731
        self.lx, self.lz = wave(nx) * self.dxi ** 2, wave(nz) * self.dzi ** 2
        self.h0 = torch.zeros((3, nz, ny, nx), **f64)

    @staticmethod
    def _lines(a, b, c, r):
        """Tridiagonal solve along dim 1; a, b, c: per row, a number or an array over the lines."""
        n = r.shape[1]
        x, h = torch.empty_like(r), [None] * n
        piv = 1.0 / b[0]
        h[0], x[:, 0] = c[0] * piv, r[:, 0] * piv
        for j in range(1, n):
            piv = 1.0 / (b[j] - h[j - 1] * a[j])
            h[j] = c[j] * piv
            x[:, j] = (r[:, j] - a[j] * x[:, j - 1]) * piv
        for j in range(n - 2, -1, -1):
            x[:, j] -= h[j] * x[:, j + 1]
        return x

    def substep(self, q, p, ns):
        ny, dt, dxi, dzi = self.ny, self.dt, self.dxi, self.dzi
        alp = self.GAM[ns] + self.ROH[ns]
        Y = lambda t: t[None, :, None]  # noqa: E731
        xp, xm = (lambda t: t.roll(-1, 2)), (lambda t: t.roll(1, 2))
        zp, zm = (lambda t: t.roll(-1, 0)), (lambda t: t.roll(1, 0))
        u, v, w = q
        df, dc = Y(self.df), Y(self.dc[:-1])
        ff, fb = Y(self.ff), Y(self.fb)
        C, P, M = slice(1, ny + 1), slice(2, ny + 2), slice(0, ny)
        fu, fw = ff * u[:, 1:] + fb * u[:, :-1], ff * w[:, 1:] + fb * w[:, :-1]  # on the faces 0..ny

        def sq(f, sh_p, sh_m, d):
            return ((sh_p(f) + f) ** 2 - (f + sh_m(f)) ** 2)[:, C] * (0.25 * d)

        vx, vz, wx, uz = v + xm(v), v + zm(v), w + xm(w), u + zm(u)
        H = [sq(u, xp, xm, dxi) + (vx[:, P] * fu[:, 1:] - vx[:, C] * fu[:, :-1]) * (0.5 * df)
             + (zp(wx) * (zp(u) + u) - wx * (u + zm(u)))[:, C] * (0.25 * dzi),
             (xp(fu) * (xp(v) + v)[:, 1:] - fu * (v + xm(v))[:, 1:])[:, :-1] * (0.5 * dxi)
             + ((v[:, P] + v[:, C]) ** 2 - (v[:, C] + v[:, M]) ** 2) * (0.25 * dc)
             + (zp(fw) * (zp(v) + v)[:, 1:] - fw * (v + zm(v))[:, 1:])[:, :-1] * (0.5 * dzi),
             (xp(uz) * (xp(w) + w) - uz * (w + xm(w)))[:, C] * (0.25 * dxi)
             + (vz[:, P] * fw[:, 1:] - vz[:, C] * fw[:, :-1]) * (0.5 * df) + sq(w, zp, zm, dzi)]
        grad = ((p - xm(p))[:, C] * dxi, (p[:, C] - p[:, M]) * dc, (p - zm(p))[:, C] * dzi)
        beta = 0.5 * alp * dt / self.ren
        lam = (1.0 + beta * self.lx)[None, None, :] * (1.0 + beta * self.lz)[:, None, None]
        new = []
        for c, f in enumerate(q):
            m, d, a = self.visc[c]
            lap = ((xp(f) - 2 * f + xm(f)) * dxi ** 2 + (zp(f) - 2 * f + zm(f)) * dzi ** 2)[:, C]
            lap = lap + f[:, P] * Y(a) + f[:, C] * Y(d) + f[:, M] * Y(m)
            r = dt * (self.ROH[ns] * self.h0[c] - self.GAM[ns] * H[c] + alp / self.ren * lap) - alp * dt * grad[c]
            self.h0[c] = -H[c]
            if c == 0:  # constant mass flux
                r = r - (r / df).sum() / (self.nx * self.nz * (1.0 / self.df).sum())
            r = torch.fft.ifft2(torch.fft.fft2(r, dim=(0, 2)) / lam, dim=(0, 2)).real
            if c == 1:
                r[:, 0] = new[0][:, 0]  # row 1 of the v lines carries the u increment
            new.append(self._lines(-beta * m, 1.0 - beta * d, -beta * a, r))
        for c, f in enumerate(q):
            j0 = 1 if c == 1 else 0
            f[:, 1 + j0:ny + 1] += new[c][:, j0:]
        div = (xp(u) - u)[:, C] * dxi + (v[:, P] - v[:, C]) * df + (zp(w) - w)[:, C] * dzi
        rhs = div / (dt * alp)
        s = torch.fft.fft(torch.fft.rfft(rhs, dim=2), dim=0)
        a, b, g = ([t[j] for j in range(ny)] for t in self.pois)
        shift = self.lx[:self.nx // 2 + 1][None, :] + self.lz[:, None]
        b = [x - shift for x in b]
        g[0] = g[0] * torch.ones_like(shift)
        g[0][0, 0], s[0, 0, 0] = 0.0, 0.0  # the mean mode's first row is pinned
        phi = torch.fft.irfft(torch.fft.ifft(self._lines(a, b, g, s), dim=0), n=self.nx, dim=2)
        u[:, C] -= (phi - xm(phi)) * (dt * alp * dxi)
        w[:, C] -= (phi - zm(phi)) * (dt * alp * dzi)
        v[:, 2:ny + 1] -= (phi[:, 1:] - phi[:, :-1]) * (dt * alp) * Y(self.dc[1:ny])
        p[:, C] += phi - beta * rhs
        p[:, 0], p[:, ny + 1] = p[:, 1], p[:, ny]


def _exact_tg(nx, ny, nz, seed, steps, ren=2800.0, dt=1e-3):
    q = list(_velocity(nx, ny, nz, seed))
    p = torch.zeros_like(q[0])
    t = _TG64(nx, ny, nz, ren, dt)
    for ns in [0] + [1, 2, 3] * steps:
        t.substep(q, p, ns)
    return dict(zip(TG_FIELDS, (*q, p)))


def _exact_stats(nx, ny, nz, seed):
    """PP_MEAN_ZX_FLOW_Xperiodic_IO: the 360 xz means of every row, as
    (ny, 360), from the cell-centred values and central differences."""
    f = _stat_fields(nx, ny, nz, seed)
    m = _TG64(nx, ny, nz, 2800.0, 1e-3, LX_IO)
    dc, dp, df = m.dc[:-1][None, :, None], m.dc[1:][None, :, None], m.df[None, :, None]
    C = slice(1, ny + 1)
    sh = lambda a, ax, n: a.roll(-n, {0: 2, 1: 1, 2: 0}[ax])  # noqa: E731  (the rows wrap only in the ghosts)
    mid = lambda a, ax: 0.5 * (a + sh(a, ax, 1))  # noqa: E731

    def diff(a, ax):
        """Central difference of a cell value."""
        if ax == 1:
            return 0.5 * ((sh(a, 1, 1) - a)[:, C] * dp + (a - sh(a, 1, -1))[:, C] * dc)
        return 0.5 * (sh(a, ax, 1) - sh(a, ax, -1))[:, C] * (m.dxi if ax == 0 else m.dzi)

    vel, flux = [f[n] for n in ("u", "v", "w")], [f[n] for n in ("gx", "gy", "gz")]
    cells = [mid(a, ax) for ax, a in enumerate(vel)]
    U, G = [a[:, C] for a in cells], [mid(a, ax)[:, C] for ax, a in enumerate(flux)]
    step = (m.dxi, df, m.dzi)
    D = [(sh(vel[i], i, 1) - vel[i])[:, C] * step[i] if i == j else diff(cells[i], j) for i in range(3) for j in range(3)]
    p, T, R, h, M, K = (f[n][:, C] for n in ("p", "t", "rho", "h", "mu", "k"))
    dh, dT = [diff(f["h"], j) for j in range(3)], [diff(f["t"], j) for j in range(3)]
    up2 = [(i, j) for i in range(3) for j in range(i, 3)]
    up3 = [(i, j, k) for i, j in up2 for k in range(j, 3)]
    terms = [(a,) for a in (*U, p, *G)] + [(a, p) for a in U]
    terms += [(U[i], U[j]) for i, j in up2] + [(U[i], G[j]) for i, j in up2]
    terms += [(U[i], U[j], U[k]) for i, j, k in up3] + [(U[i], G[j], U[k]) for i, j, k in up3]
    terms += [(a,) for a in D] + [(a, p) for a in D] + [(a, b) for a in D for b in D]
    terms += [(T,), (R,), (h,), (M,), (T, T), (R, R), (h, h), (h, R), (h, p)]
    terms += [(a, M) for a in D] + [(a, M, h) for a in D] + [(a, M, b) for a in D for b in U]
    terms += [(a, b, M) for a in D for b in D] + [(h, a) for a in U] + [(h, a) for a in G]
    terms += [(R, h, U[i], U[j]) for i, j in up2] + [(a,) for a in dh] + [(a, p) for a in dh]
    terms += [(a, K) for a in dT] + [(a, K, b) for a in dT for b in U]
    terms += [(a, K, b) for a in dT for b in D] + [(a, M, b) for a in dh for b in D]
    cols = []
    for t in terms:
        x = t[0]
        for y in t[1:]:
            x = x * y
        cols.append(x.mean(dim=(0, 2)))
    return torch.stack(cols, dim=1)


def exact(case, seed):
    """The TG steps and the statistics; the IO sections' step has no short
    restatement."""
    if case["kind"] == "stats":
        xz = _exact_stats(case["nx"], case["ny"], case["nz"], seed)
        return {"xz": xz, "xzt": xz}
    if case["kind"] == "tg":
        return _exact_tg(case["nx"], case["ny"], case["nz"], seed, case["steps"])
    if case["kind"] == "batch" and case["n"] <= 64:
        parts = [_exact_tg(c["nx"], c["ny"], c["nz"], seed + i, case["steps"], c["ren"], c["dt"])
                 for i, c in enumerate(batch64_configs(case["sizes"], case["n"]))]
        return {f: torch.cat([x[f].reshape(-1) for x in parts]) for f in TG_FIELDS}
    return None
