"""The work that a user of the library has it do, as cases that can be timed and compared.

A case is a dict of plain values.  ``kind`` says which public path it takes:

``step``      a resident ``Context`` advanced by some time steps, then its state
              read into device arrays (what a driver does between two outputs);
              ``precision`` 32 is the precision form, 64 the plain form.
``meteo``     one meteorological update of a resident context: coefficients,
              settling velocities, dry deposition and the time step.
``routines``  one class taken through a step by the fine-grained entry points
              on device arrays, as a driver that owns its arrays calls them.
``record``    the output variables of one results record.
``forecast``  a whole ``Context.run`` from host met and source series, with a
              meteorological update on the way, and its deposit maps.
``ensemble``  a ``Batch`` of scenarios of different sizes run together.

Everything is made from the seed: power-law winds with a k^-5/3 perturbation,
the standard atmosphere over a hill, a precipitation band, a grain-size
distribution over phi -2..6, a column source, and a plume of finite extent.
The precision form's results are taken as binary32, which is what it keeps.

``exact`` restates the scheme in binary64 with plain torch.
"""
import math

import numpy as np
import torch

import fall3d_gb300 as F
from fall3d_gb300 import synth

DEV = "cuda"
PI = 3.14159265358979323846
REARTH = 6356e3


# ------------------------------------------------------------------ the cases

def listed():
    def step(name, nx, ny, nz, nc, steps, precision=32, wet=True, deg=0.02):
        return dict(name=name, kind="step", nx=nx, ny=ny, nz=nz, nc=nc, steps=steps, precision=precision,
                    wet=wet, deg=deg)

    return [
        # the reduced grid of the tests, one step at a time: launches and latency
        step("step32 12x10x8x3", 12, 10, 8, 3, 1, wet=False, deg=0.05),
        # the CPU-sized workload, an operational grid of a small domain
        step("step32 80x80x25x6", 80, 80, 25, 6, 8, wet=False, deg=0.05),
        # an ensemble member's size: odd and ragged, no multiple of any tile
        step("step32 243x191x37x11", 243, 191, 37, 11, 8, deg=0.03),
        # the benchmark's forecast grid
        step("step32 400x300x50x16", 400, 300, 50, 16, 8),
        # towards the high-resolution configuration: the largest of the range
        step("step32 800x600x60x20", 800, 600, 60, 20, 3, deg=0.01),
        # the plain form on a small grid
        step("step64 32x28x14x4", 32, 28, 14, 4, 4, precision=64, deg=0.05),
        # the plain form on the benchmark's grid
        step("step64 400x300x50x16", 400, 300, 50, 16, 1, precision=64),
        # every DBS interval begins with this update
        dict(name="meteo 400x300x50x16", kind="meteo", nx=400, ny=300, nz=50, nc=16, wet=True, deg=0.02),
        # the reference's subroutines one by one, class by class
        dict(name="routines 201x149x41", kind="routines", nx=201, ny=149, nz=41, nc=1, wet=True, deg=0.03),
        # one record of the results file
        dict(name="record 400x300x50x16", kind="record", nx=400, ny=300, nz=50, nc=16, wet=True, deg=0.02),
        # a short forecast from host series, start to end
        dict(name="forecast 160x121x40x8", kind="forecast", nx=160, ny=121, nz=40, nc=8, steps=160, wet=True,
             deg=0.05),
        # members of an ensemble of different sizes advanced together
        dict(name="ensemble of 6", kind="ensemble", members=6, low=64, high=144, nz=28, nc=8, steps=120, wet=False,
             deg=0.04, sizes=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "step", "meteo", "routines", "record", "forecast", "ensemble"])
    deg = round(rng.uniform(0.01, 0.05), 4)
    wet = rng.random() < 0.5
    c = dict(kind=kind, wet=wet, deg=deg)
    if kind == "step":
        c["precision"] = rng.choice([32, 32, 32, 64])
        most = 3e8 if c["precision"] == 32 else 6e7
        while True:
            c.update(nx=_log_int(rng, 10, 900), ny=_log_int(rng, 10, 700), nz=_log_int(rng, 8, 70), nc=_log_int(rng, 3, 20))
            n = c["nx"] * c["ny"] * c["nz"] * c["nc"]
            if n <= most:
                break
        c["steps"] = rng.randint(1, max(1, min(8, int((8e8 if c["precision"] == 32 else 9e7) / n))))
    elif kind in ("meteo", "record"):
        while True:
            c.update(nx=_log_int(rng, 32, 420), ny=_log_int(rng, 28, 320), nz=_log_int(rng, 12, 60), nc=_log_int(rng, 3, 20))
            if c["nx"] * c["ny"] * c["nz"] * c["nc"] <= 9e7:
                break
    elif kind == "routines":
        c.update(nx=_log_int(rng, 20, 320), ny=_log_int(rng, 20, 240), nz=_log_int(rng, 10, 60), nc=1)
    elif kind == "forecast":
        c.update(nx=rng.randint(64, 170), ny=rng.randint(64, 130), nz=rng.randint(20, 40), nc=rng.randint(4, 10),
                 steps=rng.randint(40, 160))
    else:
        c.update(members=rng.randint(2, 6), low=64, high=rng.randint(80, 144), nz=rng.randint(20, 30),
                 nc=rng.randint(4, 8), steps=rng.randint(30, 120), sizes=rng.randint(0, 10 ** 6))
    return c


# ----------------------------------------------------------------- the inputs

def _rng(case, seed, *what):
    return np.random.default_rng([int(seed), case["nx"], case["ny"], case["nz"], *what])


def _noise(r, ny, nx, rms):
    """A field with an isotropic k^-5/3 energy spectrum of the given rms."""
    k = np.sqrt(np.fft.fftfreq(ny)[:, None] ** 2 + np.fft.fftfreq(nx)[None, :] ** 2)
    k[0, 0] = 1.0
    amp = np.sqrt(k ** (-5.0 / 3.0) / k)
    amp[0, 0] = 0.0
    f = np.real(np.fft.ifft2(amp * (r.standard_normal((ny, nx)) + 1j * r.standard_normal((ny, nx)))))
    return f * (rms / max(float(np.std(f)), 1e-30))


def _f32(a):
    """Rounded to binary32 as the DBS file holds it."""
    return a.float().double() if isinstance(a, torch.Tensor) else np.asarray(a, np.float32).astype(np.float64)


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV)


def _grid(case, seed):
    nx, ny, nz, nc, deg = (case[k] for k in ("nx", "ny", "nz", "nc", "deg"))
    r = _rng(case, seed, 0)
    lat = 37.5 + deg * (np.arange(ny) - 0.5 * (ny - 1))
    d = REARTH * (deg * PI / 180.0)
    zlayer = _f32(np.linspace(0.0, 400.0 * nz, nz))
    dz = np.empty(nz + 1)
    dz[1:nz] = np.diff(zlayer)
    dz[0], dz[nz] = dz[1], dz[nz - 1]
    Y, X = np.meshgrid(np.arange(ny) - ny // 2, np.arange(nx) - nx // 2, indexing="ij")
    hill = 1500.0 * np.exp(-(X ** 2 + Y ** 2) / (2.0 * (0.2 * min(nx, ny)) ** 2))
    phi = np.linspace(-2.0, 6.0, nc) if nc > 1 else np.array([4.0])
    diam = np.round(2.0 ** -phi, 6) / 1e3
    rhop = np.round(np.linspace(2500.0, 1000.0, nc), 1)
    sphe = np.full(nc, 0.9)
    return dict(nx=nx, ny=ny, nz=nz, nc=nc, np=nc, coord_sys=synth.COORD_LONLAT, modkv=synth.MODKV_SIMILARITY,
                modkh=synth.MODKH_RAMS, modv=synth.MODV_GANSER, wetdep=int(case["wet"]), aggregate=0, dX1=d, dX2=d,
                dx=deg, dy=deg, rkh0=0.0, rkv0=0.0, Csh=0.2275, safety_factor=0.9, vset_factor=1.0, dz=dz,
                zlayer=zlayer, Hm1=np.repeat(np.sin((90.0 - lat) * PI / 180.0)[:, None], nx, axis=1),
                topg=_f32(np.maximum(0.0, hill + _noise(r, ny, nx, 50.0))), diam=diam, rhop=rhop, sphe=sphe,
                psi=sphe.copy())


def _met(case, seed, g, snap=0):
    """The raw fields of one DBS snapshot, on the device."""
    nx, ny, nz = g["nx"], g["ny"], g["nz"]
    r = _rng(case, seed, 1 + snap)
    zl = _dev(g["zlayer"])[:, None, None]
    z = zl + _dev(g["topg"])
    t11 = 288.15 - 0.0065 * 11000.0
    T = torch.where(z <= 11000.0, 288.15 - 0.0065 * z, torch.full_like(z, t11))
    p11 = 101325.0 * (t11 / 288.15) ** (9.80665 / (287.05 * 0.0065))
    P = torch.where(z <= 11000.0, 101325.0 * (T / 288.15) ** (9.80665 / (287.05 * 0.0065)),
                    p11 * torch.exp(-9.80665 * (z - 11000.0) / (287.05 * t11)))
    T = T + _dev(_noise(r, ny, nx, 0.5))
    du, dv, dw = (_dev(_noise(r, ny, nx, s)) for s in (5.0, 5.0, 0.05))
    lift = 0.5 + 0.5 * zl / float(g["zlayer"][-1])
    m = dict(u=10.0 * (torch.clamp(zl, min=1.0) / 1000.0) ** 0.25 + du * lift, v=3.0 + dv * lift, w=dw * lift, t=T,
             tp=T * (1e5 / P) ** 0.285, rho=P / (287.05 * T))
    band = np.exp(-((np.arange(nx) / nx - 0.4 - 0.1 * snap) / 0.15) ** 2)[None, :] * np.ones((ny, 1))
    m2 = dict(ust=0.3 + 0.02 * _noise(r, ny, nx, 1.0), pblh=1000.0 + _noise(r, ny, nx, 150.0),
              rmol=_noise(r, ny, nx, 1.0 / 500.0), znt=np.full((ny, nx), 0.1), prate=5.0 * band / 3600.0,
              ldu=r.integers(1, 25, (ny, nx)).astype(np.float64))
    m = {k: _f32(v).expand(nz, ny, nx).contiguous() for k, v in m.items()}
    m.update({k: _dev(_f32(v)) for k, v in m2.items()})
    return m


def _source(case, seed, g):
    """A column of sources over the domain's centre, rates as (nsou, nc) column major."""
    nz, nc = g["nz"], g["nc"]
    n = max(1, (2 * nz) // 3)
    s = (1.0 - np.arange(n) / n) * np.exp(4.0 * (np.arange(n) / n - 1.0))
    fc = np.exp(-0.5 * ((np.arange(nc) - 0.4 * nc) / (0.25 * nc + 0.5)) ** 2)
    rate = 1e7 * _rng(case, seed, 90).uniform(0.5, 2.0) * np.outer(fc / fc.sum(), s / s.sum())
    return dict(t1=np.zeros(1, np.int32), t2=np.full(1, 10 ** 9, np.int32), nsou=np.array([n], np.int32),
                isrc=np.full(n, g["nx"] // 2 + 1, np.int32), jsrc=np.full(n, g["ny"] // 2 + 1, np.int32),
                ksrc=np.arange(1, n + 1, dtype=np.int32), tmrat=rate.reshape(-1).copy())


def _plume(case, seed, g):
    """Concentrations (nc, nz+2, ny+2, nx+2) of a plume that covers part of the domain."""
    nx, ny, nz, nc = g["nx"], g["ny"], g["nz"], g["nc"]
    r = _rng(case, seed, 91)
    c = torch.zeros((nc, nz + 2, ny + 2, nx + 2), dtype=torch.float64, device=DEV)
    x, y, z = (torch.arange(n, device=DEV, dtype=torch.float64) / n for n in (nx, ny, nz))
    for ic in range(nc):
        a, b, h, w = r.uniform(0.35, 0.65), r.uniform(0.35, 0.65), r.uniform(0.3, 0.7), r.uniform(0.1, 0.2)
        f = torch.exp(-0.5 * ((x - a) / (1.6 * w)) ** 2) * torch.exp(-0.5 * ((y - b) / w) ** 2)[:, None]
        f = f * torch.exp(-0.5 * ((z - h) / 0.2) ** 2)[:, None, None] * (1e-3 / nc)
        c[ic, 1:-1, 1:-1, 1:-1] = _f32(torch.where(f > 1e-9, f, torch.zeros_like(f)))
    return c


def _deposit(case, seed, g, which):
    ny, nx, nc = g["ny"], g["nx"], g["nc"]
    r = _rng(case, seed, 92 + which)
    f = torch.zeros((nc + 1, ny, nx), dtype=torch.float64, device=DEV)
    for ic in range(nc):
        f[ic + 1] = _dev(np.maximum(0.0, _noise(r, ny, nx, 0.1)))
    return f


def _member(case, m):
    """Member m of an ensemble case: a case of its own size."""
    r = np.random.default_rng([case["sizes"], m])
    return dict(case, kind="step", nx=int(r.integers(case["low"], case["high"] + 1)),
                ny=int(r.integers(case["low"], case["high"] + 1)), nz=int(r.integers(20, case["nz"] + 1)),
                nc=int(r.integers(4, case["nc"] + 1)))


TIMES = np.array([0, 1800, 3600], np.int32)  # snapshots every 30 minutes


def _series(case, seed, g):
    """The met series of a forecast in page-locked host memory."""
    snaps = [_met(case, seed, g, k) for k in range(len(TIMES))]

    def host(t):
        h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
        h.copy_(t)
        return h.numpy()

    met = {k: host(torch.stack([s[k] for s in snaps])) for k in snaps[0] if k != "ldu"}
    met.update(ldu=host(snaps[0]["ldu"]), times=TIMES, time_lag=0.0)
    return met


# ------------------------------------------------------------------- prepare

def _scenario(case, seed, g, met=None):
    return synth.Scenario(name=case["kind"], seed=int(seed), grid=g, met=met, src=_source(case, seed, g),
                          beg_time=0.0, end_time=float(TIMES[-1]))


def _room(s, ctx):
    """Device arrays that the context's state is read into, and its stream."""
    nx, ny, nz, nc = ctx.nx, ctx.ny, ctx.nz, ctx.nc
    new = lambda *n: torch.zeros(n, dtype=torch.float64, device=DEV)  # noqa: E731
    s.update(ctx=ctx, c=new(nc, nz + 2, ny + 2, nx + 2), cdry=new(nc + 1, ny, nx), cwet=new(nc + 1, ny, nx),
             stream=torch.cuda.ExternalStream(ctx.stream_handle()))
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        batch, members = F.Batch(8), []
        batch.set_option(F.OPT_TILE, 3)
        for m in range(case["members"]):
            mc = _member(case, m)
            g = _grid(mc, seed)
            ctx = F.Context(_scenario(mc, seed, g, _series(mc, seed, g)), F.PREC_FP32)
            members.append(_room(dict(zero=torch.zeros((g["nc"], g["nz"] + 2, g["ny"] + 2, g["nx"] + 2),
                                                       dtype=torch.float64, device=DEV)), ctx))
            members[-1]["none"] = torch.zeros((g["nc"] + 1, g["ny"], g["nx"]), dtype=torch.float64, device=DEV)
        torch.cuda.synchronize()
        return dict(case=case, batch=batch, members=members)
    g = _grid(case, seed)
    if kind == "routines":
        s = dict(case=case, g=g, **_routine_fields(case, seed, g))
        torch.cuda.synchronize()
        return s
    if kind == "forecast":
        met = _series(case, seed, g)
        ctx = F.Context(_scenario(case, seed, g, met), F.PREC_FP32)
        ctx.set_option(F.OPT_PREFETCH, 1)
        s = _room(dict(case=case, zero=torch.zeros((g["nc"], g["nz"] + 2, g["ny"] + 2, g["nx"] + 2),
                                                   dtype=torch.float64, device=DEV)), ctx)
        s["none"] = torch.zeros((g["nc"] + 1, g["ny"], g["nx"]), dtype=torch.float64, device=DEV)
        torch.cuda.synchronize()
        return s
    ctx = F.Context(_scenario(case, seed, g), F.PREC_FP32 if kind != "step" else case["precision"])
    s = dict(case=case, ctx=ctx)
    if kind == "meteo":
        s["fields"] = _met(case, seed, g)
        nx, ny, nz, nc = ctx.nx, ctx.ny, ctx.nz, ctx.nc
        s["vset"] = torch.zeros((nc, nz, ny, nx), dtype=torch.float64, device=DEV)
        s["vdep"] = torch.zeros((nc, ny, nx), dtype=torch.float64, device=DEV)
        s["coeffs"] = torch.zeros((7, nz, ny, nx), dtype=torch.float64, device=DEV)
        s["iters"] = torch.zeros((nc, nz, ny, nx), dtype=torch.int32, device=DEV)
        torch.cuda.synchronize()
        return s
    c = _plume(case, seed, g)
    if kind == "record":
        dry, wet = _deposit(case, seed, g, 0), _deposit(case, seed, g, 1)
        s["con"] = torch.zeros((ctx.nz, ctx.ny, ctx.nx), dtype=torch.float32, device=DEV)
        torch.cuda.synchronize()
        ctx.upload_state(c, dry, wet)
        return s
    m = _met(case, seed, g)
    torch.cuda.synchronize()
    ctx.meteo(fields=m)
    ctx.source(0)
    ctx.upload_state(c)
    ctx.sync()
    return _room(s, ctx)


# ----------------------------------------------------------------------- run

def _ok(rc):
    if rc:
        raise F.F3DError(rc, F.last_error())


def _state(s):
    """The context's state in the precision that it keeps: the concentrations and the classes'
    dry and wet deposits (their sum over the classes is formed with an output)."""
    ctx = s["ctx"]
    _ok(ctx.lib.f3d_download(ctx.h, *(s[k].data_ptr() for k in ("c", "cdry", "cwet")), None, None))
    if ctx.precision == 64:
        return [s["c"], s["cdry"][1:], s["cwet"][1:]]
    with torch.cuda.stream(s["stream"]):
        return [s["c"].float(), s["cdry"][1:].float(), s["cwet"][1:].float()]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "ensemble":
        slots = []
        for m in s["members"]:
            m["ctx"].upload_state(m["zero"], m["none"], m["none"])
            slots.append(s["batch"].add(m["ctx"], max_steps=case["steps"]))
        s["batch"].run()
        for slot in slots:
            s["batch"].release(slot)
        return [[*_state(m), m["ctx"].output(F.OUT_LOAD, binary32=True)] for m in s["members"]]
    if kind == "routines":
        return _run_routines(s)
    ctx = s["ctx"]
    if kind == "step":
        ctx.step(case["steps"])
        return _state(s) + [float(ctx.state()["outmass"])]
    if kind == "meteo":
        ctx.meteo(fields=s["fields"])
        _ok(ctx.lib.f3d_download(ctx.h, None, None, None, s["vset"].data_ptr(), s["vdep"].data_ptr()))
        _ok(ctx.lib.f3d_download_coeffs(ctx.h, *(f.data_ptr() for f in s["coeffs"])))
        _ok(ctx.lib.f3d_download_iters(ctx.h, s["iters"].data_ptr()))
        t = ctx.state()
        return [s["vset"], s["vdep"], s["coeffs"], np.array([t["dt"], t["dtc"]]), s["iters"]]
    if kind == "record":
        planes = [ctx.output(v, index, binary32=True)
                  for v, index in ((F.OUT_LOAD, 0), (F.OUT_WET, 0), (F.OUT_THICK, 0), (F.OUT_COL_MASS, 0),
                                   (F.OUT_PM_COL, 20), (F.OUT_C_GRND, 0), (F.OUT_PM_GRND, 20), (F.OUT_AOT05, 0))]
        _ok(ctx.lib.f3d_output(ctx.h, F.OUT_CON, 0, 0, s["con"].data_ptr(), 1))
        return planes + [s["con"]]
    ctx.run_reset()  # a new forecast on the resident grid
    ctx.upload_state(s["zero"], s["none"], s["none"])
    ctx.run(max_steps=case["steps"])
    return _state(s) + [ctx.output(F.OUT_LOAD, binary32=True), ctx.output(F.OUT_COL_MASS, binary32=True)]


def _routine_fields(case, seed, g):
    """Scaled fields of one class, as a driver holds them after its meteo update."""
    m = _met(case, seed, g)
    h = _dev(g["Hm1"])
    r = _rng(case, seed, 95)
    nz, ny, nx = g["nz"], g["ny"], g["nx"]
    zl = _dev(g["zlayer"])[:, None, None]
    f = dict(vx=m["u"] / h, vy=m["v"], vz=m["w"].clone(), rho=m["rho"] * h, zi=m["pblh"], prate=m["prate"] * 3600.0,
             vset=-(0.5 + 0.4 / m["rho"]) * torch.ones((nz, 1, 1), device=DEV, dtype=torch.float64),
             vdep=_dev(-0.01 - 0.001 * _noise(r, ny, nx, 1.0)), rkver=1.0 + 30.0 * torch.exp(-zl / 2000.0) * m["rho"],
             rkhor=(2000.0 + 500.0 * _dev(_noise(r, ny, nx, 0.3))).expand(nz, ny, nx).contiguous())
    f["vz"][0] = 0.0
    f["rkh1"] = f["rkhor"] / (h * h)
    f = {k: v.contiguous() for k, v in f.items()}
    fac = (2 * f["rkh1"] / g["dX1"] ** 2 + f["vx"].abs() / g["dX1"] + 2 * f["rkhor"] / g["dX2"] ** 2
           + f["vy"].abs() / g["dX2"] + 2 * f["rkver"] / 400.0 ** 2 + (f["vz"] + f["vset"]).abs() / 400.0)
    f.update(dt=0.5 / float(fac.max()), c=_plume(case, seed, g)[0], dz=_dev(g["dz"]), zlayer=_dev(g["zlayer"]),
             diam=_dev(g["diam"]), cdry=torch.zeros((2, ny, nx), dtype=torch.float64, device=DEV),
             cwet=torch.zeros((2, ny, nx), dtype=torch.float64, device=DEV))
    return f


def _run_routines(s):
    g, c, dt = s["g"], s["c"], s["dt"]
    n = (g["nx"], g["ny"], g["nz"], g["nz"], 1)
    F.setbcc(c, *n, s["vx"], s["vy"], s["vz"], s["vset"], s["vdep"], s["rkver"], s["dz"])
    F.advctzc(c, *n, s["vz"], s["vset"], s["dz"], dt)
    F.advctx(c, *n, s["vx"], g["dX1"], dt)
    F.advcty(c, *n, s["vy"], g["dX2"], dt)
    F.diffz(c, *n, s["dz"], dt, s["rkver"], s["rho"])
    F.diffx(c, *n, g["dX1"], dt, s["rkh1"], s["rho"])
    F.diffy(c, *n, g["dX2"], dt, s["rkhor"], s["rho"])
    F.wetdep(c, s["cwet"], 1, *n, dt, s["diam"], s["zlayer"], s["dz"], s["zi"], s["prate"])
    F.accum(c, s["cdry"], 1, *n, s["vz"], dt, s["vset"], s["vdep"])
    F.clip(c, *n[:3], 1)
    out = F.cmass2d(c, s["vx"], s["vy"], s["vz"], s["vset"], *n[:3], 1, 1, 1, 1, g["nz"], g["dX1"], g["dX2"],
                    s["dz"], dt, 0.0)
    return [c, s["cdry"], s["cwet"], float(out)]


# ---------------------------------------------------------------------- work

def work(case):
    """Bytes and operations of one pass: per step and cell of a class, c read
    and written, the settling velocity read, the seven fields that the classes
    share read once for all of them, and about 110 operations; per update, the
    six raw fields read and the coefficients, velocities and counts written,
    and about 4 drag iterations of 45 operations."""
    kind = case["kind"]
    if kind == "ensemble":
        each = [work(_member(case, m) | dict(precision=32)) for m in range(case["members"])]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    cells = case["nx"] * case["ny"] * case["nz"]
    cc = cells * case["nc"]
    size = 8 if kind == "routines" or case.get("precision") == 64 else 4
    steps = case.get("steps", 1)
    if kind == "meteo":
        return dict(bytes=8.0 * 13 * cells + 12.0 * cc, flops=180.0 * cc + 100.0 * cells)
    if kind == "record":
        return dict(bytes=4.0 * cc + 4.0 * cells + 100.0 * case["nx"] * case["ny"], flops=6.0 * cc)
    more = dict(bytes=0.0, flops=0.0) if kind != "forecast" else work(dict(case, kind="meteo"))
    return dict(bytes=steps * size * (3.0 * cc + 7.0 * cells) + 2 * more["bytes"],
                flops=steps * 110.0 * cc + 2 * more["flops"])


# --------------------------------------------------------------------- exact
# The scheme in binary64 with torch.  Concentrations are (nc, nz+2, ny+2,
# nx+2), fields (nz, ny, nx), settling velocities (nc, nz, ny, nx).

def _sign(x):
    return torch.where(torch.signbit(x) & ~torch.isnan(x), -1.0, 1.0)


def _minmod(r, l):
    return 0.5 * (_sign(r) + _sign(l)) * torch.fmin(r.abs(), l.abs())


def _bcc(c, f, vs, vdep, dz):
    """setbcc.f90"""
    vk0, vkn = f["vz"][0] + vs[:, 0], f["vz"][-1] + vs[:, -1]
    i = slice(1, -1)
    c[:, 0, i, i] = torch.where(vk0 >= 0, 0.0, c[:, 1, i, i] * (1 + dz[0] * vdep / f["rkver"][0]))
    c[:, -1, i, i] = torch.where(vkn <= 0, 0.0, c[:, -2, i, i])
    c[:, i, i, 0] = torch.where(f["vx"][:, :, 0] >= 0, 0.0, c[:, i, i, 1])
    c[:, i, i, -1] = torch.where(f["vx"][:, :, -1] <= 0, 0.0, c[:, i, i, -2])
    c[:, i, 0, i] = torch.where(f["vy"][:, 0] >= 0, 0.0, c[:, i, 1, i])
    c[:, i, -1, i] = torch.where(f["vy"][:, -1] <= 0, 0.0, c[:, i, -2, i])
    for k, a in ((0, 1), (-1, -2)):
        for y, b in ((0, 1), (-1, -2)):
            for x, d in ((0, 1), (-1, -2)):
                c[:, k, y, x] = c[:, a, b, d]


def _advance(c, v, axis, w1, w2, last):
    """The update of a sweep from work(q,1), work(q,2) and work(n+1,1)."""
    n = w1.shape[axis]
    nar = lambda a, b, e: a.narrow(axis, b, e)  # noqa: E731
    w1p = torch.cat([nar(w1, 1, n - 1), last], axis)
    w2m = torch.cat([nar(w2, 0, 1), nar(w2, 0, n - 1)], axis)
    w2p = torch.cat([nar(w2, 1, n - 1), nar(w2, n - 1, 1)], axis)
    return torch.where(v > 0, c - w1 - (w2 - w2m), c - w1p - (w2p - w2))


def _adv_z(c, f, vs, dz, dt):
    """advctzc.f90"""
    vk = f["vz"] + vs
    vm = torch.cat([vk[:, :1], vk[:, :-1]], 1)
    i = slice(1, -1)
    cm, c0, cp = c[:, :-2, i, i], c[:, 1:-1, i, i], c[:, 2:, i, i]
    d0, dm = dz[1:].reshape(-1, 1, 1), dz[:-1].reshape(-1, 1, 1)
    dzz = 2 / (d0 + dm)
    w1 = dt * (vk * c0 - vm * cm) * dzz
    v12 = (0.5 * (vk + vm)).abs()
    w2 = dt * 0.5 * dm * (1 - v12 * dt / dm) * _minmod((cp - c0) / d0, (c0 - cm) / dm) * v12 * dzz
    last = dt * vk[:, -1:] * (cp[:, -1:] - c0[:, -1:]) / dz[-1]
    c[:, 1:-1, i, i] = _advance(c0, vk, 1, w1, w2, last)


def _adv_h(c, v, axis, d, dt):
    """advctx.f90 (axis 3), advcty.f90 (axis 2)"""
    n = v.shape[axis - 1]
    inner = c[:, 1:-1, 1:-1, :] if axis == 3 else c[:, 1:-1, :, 1:-1]
    cm, c0, cp = (inner.narrow(axis, q, n) for q in (0, 1, 2))
    vm = torch.cat([v.narrow(axis - 1, 0, 1), v.narrow(axis - 1, 0, n - 1)], axis - 1)
    a = dt / d
    v12 = (0.5 * (v + vm)).abs()
    w1 = a * (v * c0 - vm * cm)
    w2 = dt * 0.5 * (1 - a * v12) * _minmod((cp - c0) / d, (c0 - cm) / d) * v12
    last = a * v.narrow(axis - 1, n - 1, 1) * (cp - c0).narrow(axis, n - 1, 1)
    c[:, 1:-1, 1:-1, 1:-1] = _advance(c0, v, axis, w1, w2, last)


def _max0(x):
    return torch.where(x > 0, x, 0.0)


def _dif_z(c, f, dz, dt):
    """diffz.f90"""
    i = slice(1, -1)
    r, K = f["rho"], f["rkver"]
    q = c[:, 1:-1, i, i] / r
    P = r * K
    d = dz.reshape(-1, 1, 1)
    grad = (q[:, 1:] - q[:, :-1]) / d[1:-1]
    face = 0.5 * (P[1:] + P[:-1]) * grad
    new = c[:, 1:-1, i, i].clone()
    new[:, 1:-1] += dt * (face[:, 1:] - face[:, :-1]) * 2 / (d[2:-1] + d[1:-2])
    low = _max0(P[0] * (q[:, 0] - c[:, 0, i, i] / r[0]) / dz[0])
    new[:, 0] += dt * (P[1] * grad[:, 0] - low) * 2 / (dz[1] + dz[0])
    top = -_max0(-(P[-1] * (c[:, -1, i, i] / r[-1] - q[:, -1]) / dz[-1]))
    new[:, -1] += dt * (top - P[-2] * grad[:, -1]) / dz[-1]
    c[:, 1:-1, i, i] = new


def _dif_h(c, rho, K, axis, d, dt):
    """diffx.f90 (axis 3), diffy.f90 (axis 2)"""
    n = rho.shape[axis - 1]
    inner = c[:, 1:-1, 1:-1, :] if axis == 3 else c[:, 1:-1, :, 1:-1]
    c0 = inner.narrow(axis, 1, n)
    P = K * rho
    q = c0 / rho
    one = lambda t, k, a=axis: t.narrow(a, k, 1)  # noqa: E731
    step = q.narrow(axis, 1, n - 1) - q.narrow(axis, 0, n - 1)
    face = 0.5 * (P.narrow(axis - 1, 1, n - 1) + P.narrow(axis - 1, 0, n - 1)) * step
    b = axis - 1
    first = _max0(one(P, 0, b) * (one(q, 0) - one(inner, 0) / one(rho, 0, b)))
    last = -_max0(-(one(P, n - 1, b) * (one(inner, n + 1) / one(rho, n - 1, b) - one(q, n - 1))))
    right = torch.cat([one(P, 1, b) * one(step, 0), face.narrow(axis, 1, n - 2), last], axis)
    left = torch.cat([first, face.narrow(axis, 0, n - 2), one(P, n - 2, b) * one(step, n - 2)], axis)
    c[:, 1:-1, 1:-1, 1:-1] = c0 + dt / (d * d) * (right - left)


def _outflow(c, f, vs, g, dz, dt):
    """cmass2d.f90"""
    ny, nx = f["vx"].shape[1:]
    fy, fx = (torch.ones(n, device=DEV, dtype=torch.float64) for n in (ny, nx))
    fy[0] = fy[-1] = fx[0] = fx[-1] = 0.5
    h = 0.5 * (dz[1:] + dz[:-1])[:, None]
    i = slice(1, -1)
    up = (fx * fy[:, None] * g["dX1"] * g["dX2"] * (f["vz"][-1] + vs[:, -1]) * c[:, -1, i, i]).sum()
    x = (fy * g["dX2"] * h * (f["vx"][:, :, -1] * c[:, i, i, -1] - f["vx"][:, :, 0] * c[:, i, i, 0])).sum()
    y = (fx * g["dX1"] * h * (f["vy"][:, -1] * c[:, i, -1, i] - f["vy"][:, 0] * c[:, i, 0, i])).sum()
    return dt * float(up + x + y)


def _step_exact(c, dry, wet, f, vs, vdep, g, dz, dt, it, diam):
    """One step of some classes in place; returns their outflow."""
    _bcc(c, f, vs, vdep, dz)
    _adv_z(c, f, vs, dz, dt)
    for axis in ((3, 2) if it % 2 == 0 else (2, 3)):
        _adv_h(c, f["vx"] if axis == 3 else f["vy"], axis, g["dX1"] if axis == 3 else g["dX2"], dt)
    _dif_z(c, f, dz, dt)
    for axis in ((3, 2) if it % 2 == 0 else (2, 3)):
        _dif_h(c, f["rho"], f["rkh1"] if axis == 3 else f["rkhor"], axis, g["dX1"] if axis == 3 else g["dX2"], dt)
    i = slice(1, -1)
    fine = diam <= 100e-6
    if g["wetdep"] and bool(fine.any()):
        lam = torch.clamp(dt * 8.4e-5 * f["prate"] ** 0.79, max=1.0)
        inside = (_dev(g["zlayer"])[:, None, None] <= f["zi"]).double()
        for ic in torch.nonzero(fine).flatten().tolist():
            wet[ic] += (inside * dz[1:].reshape(-1, 1, 1) * c[ic, i, i, i]).sum(0) * lam
            c[ic, i, i, i] *= 1 - inside * lam
    dry -= dt * c[:, 1, i, i] * torch.clamp(vs[:, 0] + vdep, max=0.0)
    c.copy_(torch.where(c > 0, c, 0.0))
    return _outflow(c, f, vs, g, dz, dt)


def _gama(diam, sphe):
    d = diam * 1e3
    lo, hi = 1e-3, 1.0
    vp = 4.0 * math.pi * (0.5 * d) ** 3 / 3.0
    ap = math.pi ** (1.0 / 3.0) * (6.0 * vp) ** (2.0 / 3.0) / sphe
    for it in range(1000):
        x = 0.5 * (lo + hi)
        e = math.acos(x)
        ao = 0.5 * math.pi * d * d * x ** (-4.0 / 3.0) * (x * x + e / math.tan(e))
        lo, hi = (lo, x) if ao < ap else (x, hi)
        if it and abs(ao - ap) < 1e-8:
            break
    return x


def _settle(T, rho, g, cd0):
    """setvset.f90 with the Ganser drag: the drag coefficient goes from cell to
    cell, heights fastest, through all classes; each cell's entry value is found
    by repeating the whole sequence until it stays."""
    nz, ny, nx = T.shape
    flat = lambda a: a.permute(2, 1, 0).reshape(-1)  # noqa: E731
    ta = float(np.float32(291.15))
    T, r = flat(T), flat(rho)
    visc = 1.827e-5 * ((ta + 120.0) / (T + 120.0)) * (T / ta) ** 1.5
    out = torch.empty((g["nc"], nz, ny, nx), dtype=torch.float64, device=DEV)
    for ic in range(g["nc"]):
        d, psi = float(g["diam"][ic]), float(g["psi"][ic])
        gam = _gama(d, float(g["sphe"][ic]))
        dnd = 0.5 * (1.0 + gam) * gam ** float(np.float32(-2.0) / np.float32(3.0))
        k1 = 1.0 / (dnd / 3.0 + 2.0 / (3.0 * math.sqrt(psi)))
        k2 = 10.0 ** (1.8148 * (-math.log10(psi)) ** 0.5743)
        num = 4.0 * 9.81 * d * float(g["rhop"][ic]) / (3.0 * r)
        b = r * d / visc * k1 * k2
        entry = torch.full_like(T, cd0)
        for sweep in range(48 if T.numel() < 7e6 else 16):  # a sweep brings the velocities some binary digits nearer
            cd, old, left = entry.clone(), torch.full_like(T, 1e5), torch.ones_like(T, dtype=torch.bool)
            for it in range(100):
                v = torch.sqrt(num / cd)
                R = b * v
                new = k2 * (24.0 / R * (1.0 + 0.1118 * R ** 0.6567) + 0.4305 / (1.0 + 3305.0 / R))
                cd = torch.where(left, new, cd)
                left &= ~((v - old).abs() <= 1e-3) if it else left
                old = v
                if not bool(left.any()):
                    break
            nxt = torch.cat([cd.new_tensor([cd0]), cd[:-1]])
            same = bool(((nxt - entry).abs() <= 1e-15 * nxt).all())
            entry = nxt
            if same:
                break
        cd0 = float(cd[-1])
        out[ic] = -torch.sqrt(num / cd).reshape(nx, ny, nz).permute(2, 1, 0)
    return out, cd0


FENG_A = [[0.0048, 0.0315, 1.2891, 1.0338], [0.0037, 0.0120, 1.3977, 1.0707], [0.0042, 0.2928, 1.3970, 0.9155],
          [0.0032, 0.1201, 1.1838, 1.0096], [0.0043, 0.1337, 1.2834, 1.1595], [0.0045, 0.0925, 1.2654, 1.0891]]
FENG_B = [[1.0, 2.7925, 2.6878, 1.2644], [1.0, 2.2413, 2.5838, 1.3247], [1.0, 3.8581, 2.5580, 1.0364],
          [1.0, 3.4407, 2.8033, 1.2069], [1.0, 3.5456, 2.7157, 1.4863], [1.0, 3.2920, 2.7227, 1.4240]]
LAND = [6, 1, 6, 6, 6, 6, 6, 6, 6, 6, 3, 6, 6, 6, 6, 6, 5, 6, 6, 3, 2, 2, 2, 2, 4]


def _dry_velocity(m, g):
    """setvdrydep.f90"""
    land = torch.tensor(LAND, device=DEV)[m["ldu"].long()] - 1
    z0, us, znt, T = float(g["zlayer"][0]), m["ust"], m["znt"], m["t"][0]
    zeta, zeta0 = m["rmol"] * z0, m["rmol"] * znt
    ra = torch.log(z0 / znt)
    e, e0 = (torch.clamp(1 - 15 * q, min=0.0) ** 0.25 for q in (zeta, zeta0))
    unstable = ra + torch.log((e0 ** 2 + 1) * (e0 + 1) ** 2 / ((e ** 2 + 1) * (e + 1) ** 2)) + 2 * (e.atan() - e0.atan())
    ra = torch.where(zeta > 0, ra + 4.7 * (zeta - zeta0), torch.where(zeta < 0, unstable, ra))
    ra = torch.where(us > 0, ra / (us * 0.4), 1e20)
    visc = 1.827e-5 * ((291.15 + 120.0) / (T + 120.0)) * (T / 291.15) ** 1.5
    re = torch.clamp(us * znt * m["rho"][0] / visc, max=40300.0)
    vd1 = 0.0226 * us * torch.exp(-0.5 * ((re - 40300.0) / 15330.0) ** 2)
    out = torch.zeros((g["nc"], *us.shape), dtype=torch.float64, device=DEV)
    for ic, d in enumerate(g["diam"]):
        if d > 100e-6:
            continue
        k = 3 if d > 10e-6 else 2 if d > 2.5e-6 else 1 if d > 0.1e-6 else 0
        a, b = (torch.tensor([row[k] for row in t], device=DEV, dtype=torch.float64)[land] for t in (FENG_A, FENG_B))
        out[ic] = -1.0 / (ra + 1.0 / (vd1 + a * us ** b))
    return out


def _central(a, axis, d):
    n = a.shape[axis]
    mid = (a.narrow(axis, 2, n - 2) - a.narrow(axis, 0, n - 2)) / (2 * d[..., 1:-1] if axis == 2 else 2 * d)
    lo = (a.narrow(axis, 1, 1) - a.narrow(axis, 0, 1)) / (d[..., :1] if axis == 2 else d)
    hi = (a.narrow(axis, n - 1, 1) - a.narrow(axis, n - 2, 1)) / (d[..., -1:] if axis == 2 else d)
    return torch.cat([lo, mid, hi], axis)


def _update(m, g, cd):
    """meteo.f90: the scaled fields, settling and deposition velocities, dt and the chain's value."""
    nz = g["nz"]
    dz, zl, h = _dev(g["dz"]), _dev(g["zlayer"])[:, None, None], _dev(g["Hm1"])
    vx, vy, vz, T, th = (m[k] for k in ("u", "v", "w", "t", "tp"))
    vz = vz.clone()
    vz[0] = 0.0
    # kappa3.f90: similarity theory in the vertical, RAMS in the horizontal
    span = (dz[2:nz] + dz[1:nz - 1]).reshape(-1, 1, 1)
    diff = lambda a: (a[2:] - a[:-2]) / span  # noqa: E731
    shear = torch.clamp(diff(vx) ** 2 + diff(vy) ** 2, min=1e-10)
    rich = 9.81 * diff(th) / (th[1:-1] * shear)
    shear, rich = (torch.cat([a, a[-1:, -1:, -1:].expand(1, *a.shape[1:])]) for a in (shear, rich))
    z = zl[1:]
    zeta = z / torch.clamp(m["pblh"], 5.0, 5e3)
    rl = m["rmol"]
    low = 0.4 * m["ust"] * z * (1 - zeta)
    low = torch.where(rl >= 0, low / (1 + 9.2 * z * rl), low * torch.sqrt(torch.clamp(1 - 13.0 * z * rl, min=0.0)))
    lc = 1 / (1 / (0.4 * z) + 1 / 30.0)
    up = lc ** 2 * torch.sqrt(shear)
    up = torch.where(rich >= 0, up / (1 + 10 * rich * (1 + 8 * rich)), up * torch.sqrt(torch.clamp(1 - 18 * rich, min=0.0)))
    rkver = torch.cat([torch.zeros_like(T[:1]), torch.where(zeta < 1, low, torch.clamp(up, min=1.0))])
    dxx = h * g["dX1"]
    uy, vx_x = _central(vx, 1, g["dX2"]), _central(vx, 2, dxx)
    vy_y, vy_x = _central(vy, 1, g["dX2"]), _central(vy, 2, dxx)
    kh = g["Csh"] ** 2 * dxx * g["dX2"] * torch.sqrt((uy + vy_x) ** 2 + 2 * (vx_x ** 2 + vy_y ** 2))
    rkhor = torch.clamp(torch.maximum(kh, 0.075 * (dxx * g["dX2"]) ** (2.0 / 3.0)), min=1e2)
    vs, cd = _settle(T, m["rho"], g, cd)
    vdep = _dry_velocity(m, g)
    # meteo.f90:108-135, corvver.f90
    topg = _dev(g["topg"])
    vx = vx / h
    zx = torch.cat([topg[:, 1:], topg[:, -1:]], 1) - topg
    zy = torch.cat([topg[1:], topg[-1:]], 0) - topg
    vz = vz - (zx / dxx * vx + zy / g["dX2"] * vy)
    f = dict(vx=vx, vy=vy, vz=vz, rho=m["rho"] * h, rkhor=rkhor, rkh1=rkhor / (h * h), rkver=rkver,
             prate=m["prate"] * 3600.0, zi=m["pblh"])
    # finddt.f90
    thin = torch.minimum(dz[:-1], dz[1:]).reshape(-1, 1, 1)
    pre = (2 * f["rkh1"] / g["dX1"] ** 2 + vx.abs() / g["dX1"] + 2 * rkhor / g["dX2"] ** 2 + vy.abs() / g["dX2"]
           + 2 * rkver / thin ** 2)
    top = 0.0
    for v in vs:
        grad = torch.cat([(v[1:2] - v[:1]) / dz[1], (v[2:] - v[:-2]) / span, (v[-1:] - v[-2:-1]) / dz[nz - 1]])
        top = max(top, float((pre + (vz + v).abs() / thin + grad.abs()).max()))
    return f, vs, vdep, 1.0 / max(top, 1e-13), cd


def _add_source(c, src, g, dt):
    """setsrc.f90"""
    n, nc = int(src["nsou"][0]), g["nc"]
    rate = src["tmrat"].reshape(nc, n)
    for s in range(n):
        i, j, k = (int(src[q][s]) for q in ("isrc", "jsrc", "ksrc"))
        h = g["Hm1"][j - 1, i - 1]
        deep = 0.5 * g["dz"][1] + g["zlayer"][0] if k == 1 else 0.5 * (g["dz"][k - 1] + g["dz"][k])
        c[:, k, j, i] += _dev(dt * rate[:, s] * h / (h * g["dX1"] * g["dX2"] * deep))


def _steps_exact(case, seed, g, c, steps, snaps, cd=1.0, times=(0,)):
    """Some steps from the state c, each snapshot's update when its time has come."""
    nc, dz, diam = g["nc"], _dev(g["dz"]), _dev(g["diam"])
    src = _source(case, seed, g)
    dry, wet = (torch.zeros((nc + 1, g["ny"], g["nx"]), dtype=torch.float64, device=DEV) for _ in range(2))
    t, gone, due = 0.0, 0.0, 0
    block = max(1, int(6e7 // (g["nx"] * g["ny"] * g["nz"])))  # classes at a time
    for it in range(1, steps + 1):
        if due < len(times) and t >= times[due]:
            f, vs, vdep, dtc, cd = _update(snaps(due), g, cd)
            dt = 0.9 * dtc
            due += 1
        t += dt
        _add_source(c, src, g, dt)
        for a in range(0, nc, block):
            b = min(nc, a + block)
            gone += _step_exact(c[a:b], dry[a + 1:b + 1], wet[a + 1:b + 1], f, vs[a:b], vdep[a:b], g, dz, dt, it,
                                diam[a:b])
    return c, dry, wet, gone


def _load(dry, wet, g):
    return (dry[1:].sum(0) + wet[1:].sum(0)) / _dev(g["Hm1"])


def _column(c, g, classes):
    w = c[classes, 1:-1, 1:-1, 1:-1].sum(0) / _dev(g["Hm1"])
    d = _dev(g["dz"])[1:-1].reshape(-1, 1, 1)
    return 1e3 * (d * 0.5 * (w[1:] + w[:-1])).sum(0)


REFF = [0.014, 0.020, 0.028, 0.040, 0.056, 0.079, 0.112, 0.158, 0.224, 0.316, 0.447, 0.631, 0.891, 1.259, 1.778, 2.512,
        3.548, 5.012, 7.079, 10.000]
QEFF = [0.00213, 0.00386, 0.00864, 0.02324, 0.06674, 0.18285, 0.44613, 0.93225, 1.63000, 2.35760, 2.83130, 2.90880,
        2.72340, 2.50530, 2.35970, 2.27100, 2.21020, 2.16410, 2.12830, 2.10050]


def _record_exact(case, seed, g):
    c, dry, wet = _plume(case, seed, g), _deposit(case, seed, g, 0), _deposit(case, seed, g, 1)
    h, every = _dev(g["Hm1"]), list(range(g["nc"]))
    pm20 = [ic for ic in every if g["diam"][ic] <= 2e-5]
    thick = 1e2 * ((dry[1:] + wet[1:]) / _dev(g["rhop"]).reshape(-1, 1, 1)).sum(0) / h
    aot = torch.zeros_like(h)
    for ic in every:
        rad = 0.5 * g["diam"][ic]
        if not REFF[0] * 1e-6 <= rad <= REFF[19] * 1e-6:
            continue
        b = 0
        for q in range(19):
            if REFF[q] * 1e-6 <= rad <= REFF[q + 1] * 1e-6:
                b = q + 1
        aot += _column(c, g, [ic]) * 1e-3 * 0.75 * QEFF[b] / (g["rhop"][ic] * (REFF[b] * 1e-6))
    ground = lambda cls: 1e3 * c[cls, 1, 1:-1, 1:-1].sum(0) / h  # noqa: E731
    return [_load(dry, wet, g), wet[1:].sum(0) / h, thick, _column(c, g, every), _column(c, g, pm20), ground(every),
            ground(pm20), aot, 1e3 * (c[:, 1:-1, 1:-1, 1:-1].sum(0) / h)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        out = []
        for m in range(case["members"]):
            mc = _member(case, m)
            g = _grid(mc, seed)
            zero = torch.zeros((g["nc"], g["nz"] + 2, g["ny"] + 2, g["nx"] + 2), dtype=torch.float64, device=DEV)
            c, dry, wet, _ = _steps_exact(mc, seed, g, zero, case["steps"], lambda k: _met(mc, seed, g, k), times=TIMES)
            out.append([c, dry[1:], wet[1:], _load(dry, wet, g)])
        return out
    g = _grid(case, seed)
    if kind == "record":
        return _record_exact(case, seed, g)
    if kind == "meteo":
        f, vs, vdep, dtc, _ = _update(_met(case, seed, g), g, 1.0)
        co = torch.stack([f[k] for k in ("vx", "vy", "vz", "rho", "rkhor", "rkh1", "rkver")])
        return [vs, vdep, co, np.array([0.9 * dtc, dtc]), None]
    if kind == "routines":
        s = _routine_fields(case, seed, g)
        c = s["c"][None].clone()
        gg = dict(g, wetdep=1)
        gone = _step_exact(c, s["cdry"][1:], s["cwet"][1:], s, s["vset"][None], s["vdep"][None], gg, s["dz"], s["dt"], 2,
                           s["diam"])
        return [c[0], s["cdry"], s["cwet"], gone]
    if kind == "forecast":
        zero = torch.zeros((g["nc"], g["nz"] + 2, g["ny"] + 2, g["nx"] + 2), dtype=torch.float64, device=DEV)
        c, dry, wet, _ = _steps_exact(case, seed, g, zero, case["steps"], lambda k: _met(case, seed, g, k), times=TIMES)
        return [c, dry[1:], wet[1:], _load(dry, wet, g), _column(c, g, list(range(g["nc"])))]
    c, dry, wet, gone = _steps_exact(case, seed, g, _plume(case, seed, g), case["steps"], lambda k: _met(case, seed, g, k))
    return [c, dry[1:], wet[1:], gone]
