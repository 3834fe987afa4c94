"""Measured cases: what a user of this framework has it compute, through its
public entry points.

Every case is one call (or, for retrievals, one request batch) on a context
that the program keeps: the control set, the emissivity tables and the
source function are set once, as the reference reads them once.  Inputs are
seeded perturbations of the standard atmosphere with the shapes of the
benchmark configurations and of the tests: 41 pressures x 30 temperatures x
320 columns per emissivity table, 2 to 300 channels, 2 to 5 emitters, 21 to
121 levels, nadir rays of about 1000 line-of-sight points (RAYDZ 0.1 km) and
limb rays of 100 to 3000.

Kinds of cases:
  formod    one observation through Context.formod (host arrays)
  dev       a batch in device memory (jgb_formod_batch_dev)
  host      a batch in host arrays through Context.formod_batch
  kernel    finite-difference Jacobians, Context.kernel_batch
  normal    K^T W K and K^T W dy on device buffers
  invert    inverses of symmetric matrices on a device buffer
  retrieve  optimal-estimation retrievals through the engine
"""
import ctypes
import math

import numpy as np
import torch

from jurassic_gb300 import native, synth
from jurassic_gb300.model import Ctl, Ret

GASES = ("CO2", "H2O", "O3", "CH4", "N2O")
TP, TT, TU = 41, 30, 320


def listed():
    return [
        # the reference's formod() on its default settings: ten limb rays of
        # one scan, three channels, double precision; a call of a few rays,
        # where the ray tracing's latency counts
        dict(name="formod limb fp64", kind="formod", view="limb", precision="fp64", nobs=1, rays=10,
             levels=81, ztop=80.0, channels=3, gases=2, ega=1, raydz=0.1, option="plain"),
        # one nadir spectrum for a data-assimilation or quick-look program:
        # brightness temperatures above an emitting surface
        dict(name="formod nadir mixed", kind="formod", view="nadir", precision="mixed", nobs=1, rays=1,
             levels=61, ztop=90.0, channels=300, gases=3, ega=1, raydz=0.1, option="bbt"),
        # simulating an orbit of nadir soundings, inputs resident (the
        # headline configuration's 100 channels, 5 emitters, 101 levels)
        dict(name="nadir batch mixed", kind="dev", view="nadir", precision="mixed", nobs=40000, rays=1,
             levels=101, ztop=100.0, channels=100, gases=5, ega=1, raydz=0.1, option="plain"),
        # the same forward model in plain double precision (reference rounding)
        dict(name="nadir batch fp64", kind="dev", view="nadir", precision="fp64", nobs=1000, rays=1,
             levels=101, ztop=100.0, channels=100, gases=5, ega=1, raydz=0.1, option="plain"),
        # limb sounder with uneven path lengths, Curtis-Godson approximation
        dict(name="limb cga mixed", kind="dev", view="limb", precision="mixed", nobs=20000, rays=1,
             levels=81, ztop=80.0, channels=32, gases=3, ega=0, raydz=0.5, option="plain"),
        # limb scans with the instrument's field of view, brightness
        # temperatures, double precision, arrays from the host
        dict(name="limb scans fov fp64", kind="host", view="limb", precision="fp64", nobs=13, rays=21,
             levels=71, ztop=90.0, channels=11, gases=4, ega=0, raydz=0.5, option="fov"),
        # nadir scenes with surface reflection, clouds and hydrostatic
        # pressures, arrays from the host
        dict(name="nadir surface mixed host", kind="host", view="nadir", precision="mixed", nobs=1500,
             rays=1, levels=77, ztop=80.0, channels=50, gases=3, ega=1, raydz=0.1, option="surface"),
        # kernel(): T and four gases on all levels, a batch of profiles
        dict(name="jacobian mixed", kind="kernel", view="nadir", precision="mixed", nobs=48, rays=1,
             levels=81, ztop=80.0, channels=150, gases=4, ega=1, raydz=0.1, option="plain"),
        # kernel() of a single profile in double precision (what the
        # reference's retrieval calls)
        dict(name="jacobian one fp64", kind="kernel", view="nadir", precision="fp64", nobs=1, rays=1,
             levels=61, ztop=80.0, channels=60, gases=3, ega=1, raydz=0.1, option="plain"),
        # normal equations of a batch of retrievals with uneven sizes
        dict(name="normal equations mixed", kind="normal", precision="mixed", nobs=512, m=150, n=405),
        # a-priori and posterior covariances: inverses of uneven sizes
        dict(name="covariance inverse", kind="invert", nobs=96, n=405),
        # a burst of retrieval requests, uneven sizes, nadir and limb mixed,
        # through the continuous-batching engine to the error analysis
        dict(name="retrievals mixed", kind="retrieve", precision="mixed", nobs=16, levels=71, channels=300),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges, no dearer than the dearest listed."""
    kind = rng.choice(("formod", "dev", "dev", "host", "kernel", "normal", "invert", "retrieve"))
    if kind == "normal":
        m, n = _log_int(rng, 20, 400), _log_int(rng, 20, 420)
        return dict(kind=kind, precision=rng.choice(("mixed", "mixed", "fp64")),
                    nobs=_log_int(rng, 1, min(1024, int(1.5e10 / (m * n * n)))), m=m, n=n)
    if kind == "invert":
        n = _log_int(rng, 20, 420)
        return dict(kind=kind, nobs=_log_int(rng, 1, min(512, int(6e9 / n ** 3))), n=n)
    if kind == "retrieve":
        return dict(kind=kind, precision="mixed", nobs=rng.randint(1, 12), levels=rng.randint(45, 95),
                    channels=300)
    view = rng.choice(("nadir", "limb"))
    precision = rng.choice(("mixed", "fp64"))
    gases, levels = rng.randint(2, 5), rng.randint(41, 121)
    ztop = float(rng.choice((70, 80, 90, 100)))
    ega = rng.choice((1, 1, 0))
    raydz = 0.1 if view == "nadir" else rng.choice((0.1, 0.25, 0.5))
    option = "plain"
    if kind in ("formod", "host"):
        option = rng.choice(("plain", "bbt", "surface") if view == "nadir" else ("plain", "bbt", "fov"))
    rays = 1 if view == "nadir" else rng.randint(3, 21) if kind != "kernel" else rng.randint(1, 3)
    channels = _log_int(rng, 2, 120)
    if kind == "formod":
        nobs = 1
    else:  # radiances of a pass, bounded by the listed cases' cost
        most = (5e4 if precision == "fp64" else 1e6) / (channels * rays)
        if kind == "kernel":
            most /= levels * (1 + gases)
        nobs = _log_int(rng, 1, max(1, min(20000, int(most))))
    return dict(kind=kind, view=view, precision=precision, nobs=nobs, rays=rays, levels=levels,
                ztop=ztop, channels=channels, gases=gases, ega=ega, raydz=raydz, option=option)


# --------------------------------------------------------------------------
# contexts: control set, tables and source function, kept by the program

_contexts = {}


def _tables(ctx, ctl):
    """Synthetic emissivity tables of the benchmark configurations' form
    (eps = 1 - exp(-k u) on log-spaced pressures and columns, rows cut to
    1e-6 <= eps <= 0.999999), computed on the GPU and handed over."""
    rng = np.random.default_rng(100 + ctl.nd)
    lib = native.load()
    ctx._check(lib.jgb_tables_init(ctx.h, TP, TT, TU))
    pg = np.logspace(-3, math.log10(1100.0), TP)
    ug = np.logspace(10, 26, TU)
    tg = np.broadcast_to(np.linspace(180.0, 320.0, TT), (TP, TT))
    d = dict(dtype=torch.float64, device="cuda")
    shape = torch.tensor(pg / 1013.0, **d)[:, None].log(), torch.tensor(tg / 250.0, **d).log()
    u64 = torch.tensor(ug, **d)
    u32 = u64.float().expand(TP, TT, TU)
    nt = np.full(TP, TT, np.int32)
    p, t = np.ascontiguousarray(pg), np.ascontiguousarray(tg)
    for ig, name in enumerate(ctl.emitter):
        col = synth._COLUMNS[name]
        lo, hi = max(0.01 / col, 1.5e-25), min(100.0 / col, 1e-17)
        k0 = np.exp(rng.uniform(np.log(min(lo, hi / 10)), np.log(hi), ctl.nd))
        a, b = rng.uniform(0.0, 0.5, ctl.nd), rng.uniform(-1.0, 1.0, ctl.nd)
        for i in range(ctl.nd):
            k = k0[i] * torch.exp(a[i] * shape[0] + b[i] * shape[1])
            eps = (-torch.expm1(-k[:, :, None] * u64)).float()
            keep = (eps >= 1e-6) & (eps <= 0.999999)
            keep[:, :, 1:] &= eps[:, :, 1:] > eps[:, :, :-1]
            order = torch.argsort((~keep).to(torch.uint8), dim=2, stable=True)
            n = keep.sum(2)
            valid = torch.arange(TU, device="cuda") < n[:, :, None]
            e = torch.where(valid, eps.gather(2, order), 0.0).cpu().numpy()
            u = torch.where(valid, u32.gather(2, order), 0.0).cpu().numpy()
            n = n.to(torch.int32).cpu().numpy()
            f = lambda v, c: v.ctypes.data_as(ctypes.POINTER(c))  # noqa: E731
            ctx._check(lib.jgb_set_table(ctx.h, i, ig, TP, f(p, ctypes.c_double), f(nt, ctypes.c_int),
                                         f(t, ctypes.c_double), f(n, ctypes.c_int),
                                         f(u, ctypes.c_float), f(e, ctypes.c_float), TT, TU))


def _context(case):
    key = tuple((k, case.get(k)) for k in ("kind", "channels", "gases", "ega", "raydz", "option", "ztop"))
    if key in _contexts:
        _contexts[key] = _contexts.pop(key)  # the most recently used last
        return _contexts[key]
    kind, option = case["kind"], case.get("option", "plain")
    nd = case.get("channels", 2)
    if kind == "retrieve":
        emitter = ["CO2", "H2O", "O3"]
    else:
        emitter = list(GASES[:case.get("gases", 2)])
    ctl = Ctl(emitter=emitter, nu=np.linspace(650.0, 2400.0, nd), formod=case.get("ega", 1),
              raydz=case.get("raydz", 0.1), write_bbt=int(option in ("bbt", "fov")))
    if option == "bbt":
        ctl.sfnu, ctl.sftype = np.array([600.0, 2500.0]), 1
    if option == "surface":
        ctl.sfnu, ctl.sftype = np.array([600.0, 1200.0, 2500.0]), 2
        ctl.clnu, ctl.hydz = np.array([600.0, 2500.0]), 0.0
    if kind == "kernel":
        ctl.rett_zmin, ctl.rett_zmax = 0.0, case["ztop"]
        ctl.retq_zmin, ctl.retq_zmax = np.zeros(ctl.ng), np.full(ctl.ng, case["ztop"])
    if kind == "retrieve":
        ctl.rett_zmin, ctl.rett_zmax = 0.0, 60.0
        ctl.retq_zmin, ctl.retq_zmax = np.array([-999.0, 0.0, -999.0]), np.array([-999.0, 20.0, -999.0])
    ctx = native.Context(ctl)
    if kind not in ("normal", "invert"):
        _tables(ctx, ctl)
        ctx.set_filters(synth.make_filters(ctl))
    if option == "fov":
        dz = np.linspace(-1.8, 1.8, 13)
        ctx.set_fov(dz, 1.0 - np.abs(dz) / 2.0)
    while len(_contexts) >= 3:
        _contexts.pop(next(iter(_contexts)))
    _contexts[key] = (ctx, ctl)
    return ctx, ctl


# --------------------------------------------------------------------------
# inputs


def _batch(case, ctl, seed):
    """Seeded perturbations of the standard atmosphere: a temperature offset
    and wave (+-5 K together), gas factors (+-20 %), one profile and scan per
    observation, as numpy arrays in the library's batch layout."""
    rng = np.random.default_rng(seed)
    nobs, nr, nl = case["nobs"], case["rays"], case["levels"]
    z = np.linspace(0.0, case["ztop"], nl)
    t0 = synth.std_temperature(z)
    p0 = synth.hydrostatic_pressure(z, t0)
    q0 = np.stack([synth.std_vmr(e, z) for e in ctl.emitter])
    col = lambda lo, hi: rng.uniform(lo, hi, (nobs, 1))  # noqa: E731
    t = t0 + col(-2.5, 2.5) + col(-2.5, 2.5) * np.sin(z / 15.0 + col(0, 6.3))
    q = q0[:, None, :] * (1 + rng.uniform(-0.2, 0.2, (ctl.ng, nobs, 1)))
    lat, lon = rng.uniform(-60, 60, nobs), rng.uniform(-180, 180, nobs)
    L, R = nobs * nl, nobs * nr
    scal = np.zeros((nobs, 5 + ctl.ncl + ctl.nsf))
    if ctl.ncl:  # a thin cloud layer
        scal[:, 0], scal[:, 1] = rng.uniform(4, 12, nobs), rng.uniform(0.3, 1.0, nobs)
        scal[:, 2:2 + ctl.ncl] = rng.uniform(1e-3, 5e-2, (nobs, ctl.ncl))
    if ctl.nsf:  # surface temperature and emissivities
        scal[:, 4 + ctl.ncl] = 288.0 + rng.uniform(-8, 8, nobs)
        scal[:, 5 + ctl.ncl:] = rng.uniform(0.85, 0.99, (nobs, ctl.nsf))
    time = np.arange(nobs, dtype=np.float64)
    rep = lambda v: np.repeat(v, nr)  # noqa: E731
    if case["view"] == "nadir":
        geo = np.stack([rep(time), np.full(R, 705.0), rep(lon), rep(lat), np.zeros(R), rep(lon),
                        rep(lat) + rng.uniform(-3, 3, R)])
    else:
        zt = np.sort(rng.uniform(5.0, 60.0, (nobs, nr)), axis=1).reshape(-1)
        geo = np.stack([rep(time), np.full(R, 800.0), rep(lon), rep(lat), zt, rep(lon),
                        rep(lat) + synth.limb_vplat(zt, 800.0)])
    return synth.Batch(
        nobs=nobs, lev_off=(np.arange(nobs + 1) * nl).astype(np.int32), time=np.repeat(time, nl),
        z=np.tile(z, nobs), lon=np.repeat(lon, nl), lat=np.repeat(lat, nl), p=np.tile(p0, nobs),
        t=t.reshape(-1), q=np.ascontiguousarray(q.reshape(ctl.ng, L)), k=np.zeros((ctl.nw, L)),
        scal=scal, ray_off=(np.arange(nobs + 1) * nr).astype(np.int32), geo=geo,
        rad=np.zeros((ctl.nd, R)), tau=np.zeros((ctl.nd, R)), tp=np.zeros((3, R)))


def _sizes(case):
    """Uneven problem sizes (the same for every seed): half of them at the
    case's own, the others down to a fifth of it."""
    rng = np.random.default_rng(case["nobs"])
    out = []
    for key in ("m", "n"):
        if key in case:
            f = np.where(rng.random(case["nobs"]) < 0.5, 1.0, rng.uniform(0.2, 1.0, case["nobs"]))
            out.append(np.maximum(1, (f * case[key]).astype(np.int32)))
    return out


def _requests(case, ctx, ctl, seed):
    """Retrieval requests: the standard atmosphere as a priori, measurements
    of a perturbed one with 0.2 % noise.  Levels (0-100 km), measured
    channels (the others NaN) and the nadir or limb view are uneven, the
    same for every seed."""
    size, rng = np.random.default_rng(case["nobs"]), np.random.default_rng(seed)
    apr, truth = [], []
    for i in range(case["nobs"]):
        z = np.linspace(0.0, 100.0, int(size.integers(case["levels"] - 25, case["levels"] + 26)))
        lat, lon = float(rng.uniform(-60, 60)), float(rng.uniform(-180, 180))
        at = dict(nw=ctl.nw, time=float(i), lon=lon, lat=lat)
        obs = synth.nadir_obs(ctl.nd, [lat], time=float(i), lon=lon) if i % 2 == 0 else synth.limb_obs(
            ctl.nd, np.sort(rng.uniform(8.0, 30.0, 5)), time=float(i), lon=lon, lat=lat)
        apr.append((synth.profile(ctl.emitter, z, **at), obs))
        truth.append((synth.profile(ctl.emitter, z, dt=float(rng.uniform(-3, 3)),
                                    dq=1 + rng.uniform(-0.2, 0.2, ctl.ng), **at), obs))
    rad = ctx.formod_batch(synth.pack(ctl, truth), native.FP64).rad
    rad = rad * (1 + 2e-3 * rng.standard_normal(rad.shape))
    b = synth.pack(ctl, apr)
    for i in range(case["nobs"]):
        rad[int(size.integers(50, ctl.nd + 1)):, b.ray_off[i]:b.ray_off[i + 1]] = np.nan
    b.rad = rad
    return b


def prepare(case, seed):
    ctx, ctl = _context(case)
    kind = case["kind"]
    prec = native.MIXED if case.get("precision") == "mixed" else native.FP64
    s = dict(kind=kind, ctx=ctx, ctl=ctl, prec=prec)
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda n: torch.randn(int(n), dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    if kind == "normal":
        m, n = _sizes(case)
        s.update(m=m, n=n)
        # Jacobian-like columns: magnitudes over three decades
        cols = torch.cat([torch.exp(-7.0 * torch.linspace(0, 1, int(v), dtype=torch.float64, device="cuda"))
                          .expand(int(u), int(v)).reshape(-1) for u, v in zip(m, n)])
        s["K"] = rand((m.astype(np.int64) * n).sum()) * cols
        s["w"] = 0.5 + rand(m.sum()).abs()
        s["dy"] = rand(m.sum())
        s["A"] = torch.zeros(int((n.astype(np.int64) ** 2).sum()), dtype=torch.float64, device="cuda")
        s["b"] = torch.zeros(int(n.sum()), dtype=torch.float64, device="cuda")
    elif kind == "invert":
        (n,) = _sizes(case)
        blocks = []
        for i, v in enumerate(n):
            v = int(v)
            if i % 2 == 0:  # a-priori covariance: exponential correlation along the levels
                z = torch.linspace(0, 60, v, dtype=torch.float64, device="cuda")
                sd = 1.5 + 0.3 * rand(v).clamp(-3, 3)
                blocks.append(sd[:, None] * sd[None, :] * torch.exp(-(z[:, None] - z[None, :]).abs() / 3.0))
            else:           # a Gauss-Newton matrix S_a^-1 + K^T W K
                x = rand(v * v).reshape(v, v)
                blocks.append(x @ x.T / v + 0.5 * torch.eye(v, dtype=torch.float64, device="cuda"))
        s.update(n=n, A=torch.cat([b.reshape(-1) for b in blocks]))
    elif kind == "retrieve":
        b = _requests(case, ctx, ctl, seed)
        # observation files carry six significant digits
        scale = 10.0 ** (np.floor(np.log10(np.abs(b.rad))) - 5)
        b.rad = np.round(b.rad / scale) * scale
        ret = Ret(kernel_recomp=1, conv_itmax=10, conv_dmin=0.1, err_ana=1,
                  err_noise=np.full(ctl.nd, 1e-4), err_formod=np.full(ctl.nd, 0.5), err_temp=2.0,
                  err_temp_cz=3.0, err_temp_ch=-999.0, err_q=np.array([0.0, 30.0, 0.0]),
                  err_q_cz=np.array([-999.0, 3.0, -999.0]), err_q_ch=np.full(3, -999.0))
        s.update(batch=b, engine=ctx.engine(ret, prec))
    else:
        b = _batch(case, ctl, seed)
        if kind == "formod":
            s["atm"], s["obs"] = b.item(ctl, 0)
        elif kind == "dev":
            s["dev"] = {k: torch.from_numpy(getattr(b, k)).cuda() for k in
                        ("lev_off", "time", "z", "lon", "lat", "p", "t", "q", "k", "scal", "ray_off",
                         "geo", "rad", "tau", "tp")}
            s["ptrs"] = {k: v.data_ptr() for k, v in s["dev"].items()}
            s["nobs"] = b.nobs
        else:
            s["batch"] = b
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------------
# one pass


def _void(t):
    return ctypes.c_void_p(t.data_ptr())


def _ints(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_int))


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "formod":
        o = ctx.formod(s["atm"], s["obs"], s["prec"])
        return dict(rad=o.rad, tau=o.tau, tpz=o.tpz, tplon=o.tplon, tplat=o.tplat)
    if kind == "dev":
        ctx.formod_batch_ptrs(s["ptrs"], s["nobs"], s["prec"])
        return {k: s["dev"][k] for k in ("rad", "tau", "tp")}
    if kind == "host":
        o = ctx.formod_batch(s["batch"], s["prec"])
        return dict(rad=o.rad, tau=o.tau, tp=o.tp, p=o.p)
    if kind == "kernel":
        K, o = ctx.kernel_batch(s["batch"], s["prec"])
        return dict(K=np.concatenate([k.reshape(-1) for k in K]) if len(K) > 1 else K[0].reshape(-1),
                    rad=o.rad, tau=o.tau)
    if kind == "normal":
        ctx._check(native.load().jgb_normal_equations_dev(
            ctx.h, len(s["m"]), _ints(s["m"]), _ints(s["n"]), _void(s["K"]), _void(s["w"]),
            _void(s["dy"]), _void(s["A"]), _void(s["b"]), s["prec"], None))
        return dict(A=s["A"], b=s["b"])
    if kind == "invert":
        A = s["A"].clone()
        torch.cuda.current_stream().synchronize()  # the call runs on its own stream
        st = np.zeros(len(s["n"]), np.int32)
        ctx._check(native.load().jgb_matrix_invert_dev(ctx.h, len(s["n"]), _ints(s["n"]), _void(A),
                                                       _ints(st), None))
        return dict(A=A, status=st)
    res = s["engine"].run(s["batch"])
    cat = lambda k: np.concatenate([np.ravel(r[k]) for r in res])  # noqa: E731
    most = s["engine"].r.conv_itmax + 1  # the costs' histories end with the iterations
    costs = np.stack([np.pad(r["costs"], (0, most - len(r["costs"]))) for r in res])
    return dict({k: cat(k) for k in ("x", "rad", "tau", "tp", "cov", "avk", "err_total",
                                     "err_noise", "err_formod", "cont", "res")},
                costs=costs, iters=np.array([r["iters"] for r in res]), status=np.array([r["status"] for r in res]))


# --------------------------------------------------------------------------
# work and exact values


def _points(case):
    """Line-of-sight points of a ray: one per RAYDZ of altitude, down and up
    again in the limb (tangent heights 5 to 60 km), steps of at most 10 km."""
    if case["view"] == "nadir":
        return case["ztop"] / case["raydz"]
    return 2 * (case["ztop"] - 32.0) / case["raydz"] + 30


def work(case):
    """Bytes: inputs, outputs and the emissivity tables' entries once (or, for
    small calls, the eight entries that each lookup interpolates between).
    Flops: an interpolation in the tables of every (point, channel, emitter),
    or the products."""
    kind = case["kind"]
    if kind == "normal":
        f = 0.64  # mean of the products of the uneven sizes
        m, n, k = case["m"], case["n"], case["nobs"] * f
        return {"bytes": 8.0 * k * (m * n + n * n + 2 * m + n), "flops": 1.0 * k * m * n * (n + 2)}
    if kind == "invert":
        n, k = case["n"], case["nobs"] * 0.66
        return {"bytes": 16.0 * k * n * n, "flops": 1.0 * k * n ** 3}
    if kind == "retrieve":  # three iterations, each with a Jacobian and two forward models
        nl, nd, ng, rays = case["levels"], case["channels"] * 0.58, 3, 3
        state = nl * 0.8
        nrad = case["nobs"] * rays * nd * 3 * (state + 2)
        pts = 1200
        tables = case["channels"] * ng * TP * TT * TU * 8.0
        return {"bytes": tables + case["nobs"] * 8.0 * (state * state * 3 + nl * 9),
                "flops": nrad * pts * (ng * 60.0 + 30.0)}
    nd, ng, nl = case["channels"], case["gases"], case["levels"]
    rays = case["nobs"] * case["rays"]
    runs = 1
    out = rays * nd * 16.0
    if kind == "kernel":
        runs += nl * (1 + ng)
        out += rays * nd * nl * (1 + ng) * 8.0
    steps = rays * runs * _points(case) * nd * ng
    tables = min(nd * ng * TP * TT * TU * 8.0, steps * 64.0)
    return {"bytes": tables + out + 8.0 * case["nobs"] * nl * (6 + ng) + rays * 56.0,
            "flops": steps * 60.0 + steps / ng * 30.0}


def exact(case, seed):
    """Normal equations and inverses in 64 bits.  The forward model, its
    Jacobians and the retrievals have no value here: they would take a
    restatement of the whole radiative-transfer model."""
    if case["kind"] not in ("normal", "invert"):
        return None
    s = prepare(case, seed)
    off = 0
    if case["kind"] == "invert":
        out = []
        for v in s["n"]:
            v = int(v)
            inv = torch.linalg.inv(s["A"][off:off + v * v].reshape(v, v))
            out.append((0.5 * (inv + inv.T)).reshape(-1))
            off += v * v
        return dict(A=torch.cat(out), status=None)
    A, b, om = [], [], 0
    for m, n in zip(s["m"], s["n"]):
        m, n = int(m), int(n)
        w = s["w"][om:om + m]
        K = s["K"][off:off + m * n].reshape(m, n) * w[:, None]
        A.append((K.T @ K).reshape(-1))
        b.append(K.T @ (w * s["dy"][om:om + m]))
        off += m * n
        om += m
    return dict(A=torch.cat(A), b=torch.cat(b))
