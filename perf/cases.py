"""Performance cases: the work that a host model has this framework do, through its public entry points.

Each family stands for one use of the library (the comments in listed() say which):

  step         getm_time_loop over one macro step (M micro steps and one integrate_3d), or, with
               runtype 1, over M micro steps of the barotropic model: closed irregular domain
               ('islands') or shelf with a tide on its western open boundary ('shelf'); plain FP64
               or the mixed FP32/FP64 step
  tracer       getm_tracer_step: split advection and implicit vertical diffusion of one tracer
  gradient     getm_tracer_gradient: the checkpointed adjoint of a run of tracer steps
  density      getm_do_eqstate and getm_internal_pressure on a model state
  tridiagonal  getm_tridiagonal_columns: the column solver on a host's own coefficients

Inputs are seeded and made on the GPU. exact() restates every path in plain 64-bit torch.
"""
from __future__ import annotations

import math

import torch

from code_b200 import state as S
from code_b200.getm import HALFSPLIT, MUSCL, P2, P2_PDM, SUPERBEE, UPSTREAM, BcDevice, Context
from code_b200.grid import Grid

DTYPES = {"f64": torch.float64, "f32": torch.float32, "mixed": torch.float32}


# --------------------------------------------------------------------------------------------------
# the cases
def _step(name, nx, ny, kmax, dtype, recipe, runtype=4, M=20):
    return dict(name=name, family="step", nx=nx, ny=ny, kmax=kmax, dtype=dtype, recipe=recipe, runtype=runtype, M=M)


def _tracer(name, nx, ny, kmax, dtype, scheme, land, AH=0.0):
    return dict(name=name, family="tracer", nx=nx, ny=ny, kmax=kmax, dtype=dtype, scheme=scheme, land=land, AH=AH)


def listed():
    return [
        # a harbour or estuary run of the depth-averaged model: 20 micro steps with a tide; every
        # launch is small, so the launches themselves count
        _step("barotropic_128x96_f64", 128, 96, 4, "f64", "shelf", runtype=1),
        # one passive tracer of a small study domain (the 128x128x20 tracer configuration)
        _tracer("tracer_128x128x20_f64", 128, 128, 20, "f64", SUPERBEE, 0.0),
        # a biogeochemical tracer in FP32 on a domain of odd size with islands
        _tracer("tracer_701x555x33_f32", 701, 555, 33, "f32", P2_PDM, 0.3),
        # the same work in FP64 on a large domain
        _tracer("tracer_1024x1024x40_f64", 1024, 1024, 40, "f64", P2_PDM, 0.3),
        # the tidal-shelf configuration, both precisions: open boundary, so the separate
        # sealevel / boundary / depth launches
        _step("tidal_shelf_512x512x30_f64", 512, 512, 30, "f64", "shelf"),
        _step("tidal_shelf_512x512x30_mixed", 512, 512, 30, "mixed", "shelf"),
        # a small regional model of odd size: the layouts without 16-byte aligned rows
        _step("islands_259x193x25_mixed", 259, 193, 25, "mixed", "islands"),
        # the irregular domain in plain FP64 (a quarter of the benchmark's area) and the benchmark's
        # own mixed-precision step
        _step("islands_1024x1024x50_f64", 1024, 1024, 50, "f64", "islands"),
        _step("islands_2048x2048x50_mixed", 2048, 2048, 50, "mixed", "islands"),
        # the tracer-adjoint configuration's domain: ten steps, checkpoints every five
        dict(name="gradient_256x256x30_f64", family="gradient", nx=256, ny=256, kmax=30, dtype="f64",
             scheme=SUPERBEE, land=0.0, AH=0.0, nsteps=10, every=5),
        # a host that keeps its own time loop and asks for density, buoyancy and pressure gradients
        dict(name="density_1024x1024x40_mixed", family="density", nx=1024, ny=1024, kmax=40, dtype="mixed",
             recipe="islands", eos=1),
        # a host's own implicit column equations, 512 x 512 columns of 40 levels
        dict(name="tridiagonal_262144x40_f64", family="tridiagonal", ncol=512 * 512, kmax=40),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed families: sizes over their whole ranges, odd ones among them."""
    fam = rng.choice(("step", "step", "step", "tracer", "tracer", "tracer", "gradient", "density", "tridiagonal"))
    if fam == "tridiagonal":
        return dict(family=fam, ncol=_log_int(rng, 2000, 500000), kmax=rng.randint(6, 60))
    nx, ny = _log_int(rng, 48, 1100), _log_int(rng, 48, 1100)
    kmax = rng.randint(6, 50)
    if fam == "gradient":
        return dict(family=fam, nx=_log_int(rng, 48, 256), ny=_log_int(rng, 48, 256), kmax=rng.randint(6, 30),
                    dtype=rng.choice(("f64", "f32")), scheme=rng.choice((P2, MUSCL, SUPERBEE, P2_PDM)),
                    land=rng.choice((0.0, 0.3)), AH=0.0, nsteps=rng.randint(4, 10), every=rng.randint(2, 5))
    if fam == "tracer":
        return dict(family=fam, nx=nx, ny=ny, kmax=kmax, dtype=rng.choice(("f64", "f32")),
                    scheme=rng.choice((UPSTREAM, P2, MUSCL, SUPERBEE, P2_PDM, P2_PDM)),
                    land=rng.choice((0.0, 0.3)), AH=rng.choice((0.0, 0.0, 20.0)))
    if fam == "density":
        return dict(family=fam, nx=nx, ny=ny, kmax=kmax, dtype=rng.choice(("f64", "mixed")),
                    recipe=rng.choice(("shelf", "islands")), eos=rng.choice((1, 1, 2)))
    return dict(family=fam, nx=nx, ny=ny, kmax=kmax, dtype=rng.choice(("f64", "mixed")),
                recipe=rng.choice(("shelf", "islands")), runtype=rng.choice((4, 4, 4, 1)),
                M=rng.choice((10, 20, 30)))


def work(case):
    """Bytes and operations one pass cannot do without: every input read once, every output written
    once (3D fields of the case's type, 2D fields FP64)."""
    if case["family"] == "tridiagonal":
        n = case["ncol"] * (case["kmax"] + 1)
        return {"bytes": 5 * 8 * n, "flops": 8 * n}
    wb = 8 if case["dtype"] == "f64" else 4
    n2 = case["nx"] * case["ny"]
    n = n2 * case["kmax"]
    if case["family"] == "tracer":
        return {"bytes": 10 * wb * n, "flops": 260 * n}  # f, uu, vv, ww, hu, hv, ho, hn, nuh; f
    if case["family"] == "gradient":
        return {"bytes": 14 * wb * n, "flops": 700 * n * case["nsteps"]}
    if case["family"] == "density":
        return {"bytes": 9 * wb * n, "flops": 40 * n}  # T, S, hn, hun, hvn; rho, buoy, idpdx, idpdy
    micro = 380 * n2 * case["M"]
    if case["runtype"] == 1:
        return {"bytes": 8 * n2 * 50, "flops": micro}
    # read uu, vv, T, S, num, nuh, buoy, hun, hvn (and the carried errors); written: the velocities
    # and their advection, the six heights, the pressure gradients, T, S, rho, buoy
    words = 9 + 17
    extra = 8 * n if case["dtype"] == "mixed" else 0
    return {"bytes": words * wb * n + extra + 8 * n2 * 90, "flops": 1100 * n + micro}


# --------------------------------------------------------------------------------------------------
# inputs
def _gen(device, seed):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _randn(gen, *shape):
    return torch.randn(shape, generator=gen, device=gen.device, dtype=torch.float64)


def _smooth(gen, ny, nx, sigma):
    """Gaussian-smoothed unit noise of an ny x nx plane."""
    k1 = torch.fft.fftfreq(nx, device=gen.device, dtype=torch.float64)[None, :]
    k2 = torch.fft.fftfreq(ny, device=gen.device, dtype=torch.float64)[:, None]
    f = torch.fft.ifft2(torch.fft.fft2(_randn(gen, ny, nx)) *
                        torch.exp(-2 * (math.pi * sigma) ** 2 * (k1 ** 2 + k2 ** 2))).real
    return (f - f.mean()) / f.std()


def _sh(a, di, dj):
    """a at (i+di, j+dj): the last two axes shifted, zero outside the plane."""
    nj, ni = a.shape[-2:]
    out = torch.zeros_like(a)
    out[..., max(0, -dj):nj - max(0, dj), max(0, -di):ni - max(0, di)] = \
        a[..., max(0, dj):nj - max(0, -dj), max(0, di):ni - max(0, -di)]
    return out


def _masks(az):
    """au, av, ax of the haloed plane from az (0 land, 1 water, 2 open boundary)."""
    def pair(a, b):
        both = (a > 0) & (b > 0)
        return torch.where(both, a + b - 1, torch.zeros_like(a))
    e, n = _sh(az, 1, 0), _sh(az, 0, 1)
    au, av = pair(az, e), pair(az, n)
    ax = ((az >= 1) & (e >= 1) & (n >= 1) & (_sh(az, 1, 1) >= 1)).to(az.dtype)
    return au, av, ax


def _bathymetry(recipe, gen, g, land, hmin=5.0, hmax=150.0):
    """(az, H) of the haloed plane: 'shelf' 10-200 m across i, 'islands' smoothed noise with the
    fraction `land` of it dry, 'flat' 20 m."""
    ny, nx, dev = g.ny, g.nx, gen.device
    az = torch.zeros(g.shape2(), dtype=torch.int32, device=dev)
    H = torch.zeros(g.shape2(), dtype=torch.float64, device=dev)
    inner = (slice(2, 2 + ny), slice(2, 2 + nx))
    if recipe == "islands" and land > 0:
        f = _smooth(gen, ny, nx, max(2.0, 40.0 * nx / 2048.0))
        p = torch.sort(f.reshape(-1))[0][int(land * f.numel())]
        wet = f >= p
        H[inner] = torch.where(wet, hmin + (hmax - hmin) * (f - p) / (f.max() - p), torch.zeros_like(f))
        az[inner] = wet.to(torch.int32)
    else:
        x = (torch.arange(nx, device=dev, dtype=torch.float64) + 0.5) - nx / 2
        row = 20.0 + 0 * x if recipe == "flat" else 10.0 + 95.0 * (1.0 + torch.tanh(x / max(4.0, min(20.0, nx / 8))))
        H[inner] = row[None, :].expand(ny, nx)
        az[inner] = 1
    for d in (1, 0):  # the halo repeats the edge lines
        H[:, d], H[:, -1 - d] = H[:, d + 1], H[:, -2 - d]
        H[d, :], H[-1 - d, :] = H[d + 1, :], H[-2 - d, :]
    return az, H


def _flow(gen, g, H, au, av, umax=0.3):
    """Depth-integrated transports (U, V) along the contours of a random streamfunction that
    vanishes at the coasts and the walls, with speeds up to umax."""
    ny, nx, dev = g.ny, g.nx, gen.device
    inner = (slice(2, 2 + ny), slice(2, 2 + nx))
    ramp = lambda n: torch.sin(math.pi * (torch.arange(n, device=dev, dtype=torch.float64) + 1) / (n + 1))  # noqa: E731
    psi = torch.zeros_like(H)  # at the X points; the coasts of the irregular domain are 5 m deep
    psi[inner] = (_smooth(gen, ny, nx, max(3.0, nx / 20.0)) + 0.2) * torch.clamp(H[inner] - 5.0, min=0.0) \
        * ramp(ny)[:, None] * ramp(nx)[None, :]
    U = -(psi - _sh(psi, 0, -1)) * (au > 0)
    V = (psi - _sh(psi, -1, 0)) * (av > 0)
    one = torch.ones((), dtype=torch.float64, device=dev)
    HU, HV = 0.5 * (H + _sh(H, 1, 0)), 0.5 * (H + _sh(H, 0, 1))
    speed = torch.maximum((U.abs() / torch.where(HU > 0, HU, one)).max(), (V.abs() / torch.where(HV > 0, HV, one)).max())
    return U * umax / speed, V * umax / speed


def _state(case, seed, device="cuda"):
    """A model state under way: (grid, tensors, real and integer parameters, open boundaries)."""
    shelf = case["recipe"] == "shelf"
    M = case.get("M", 20)
    dt = 3.0 * M
    g = Grid(case["nx"], case["ny"], case["kmax"], 1000.0, 1000.0)
    kmax = g.kmax
    gen = _gen(device, seed)
    az, H = _bathymetry(case["recipe"], gen, g, 0.0 if shelf else 0.3)
    bdy = None
    if shelf:  # an M2 tide of half a metre, clamped on the western side
        az[2:2 + g.ny, 2] = 2
        bdy = S.OpenBoundaries(west=[(g.imin, g.jmin, g.jmax, S.CLAMPED)], ramp=40, amp=0.5, phase=0.3, period=44712.0)
    au, av, ax = _masks(az)
    zero2 = lambda: torch.zeros(g.shape2(), dtype=torch.float64, device=device)  # noqa: E731
    f2 = {n: zero2() for n in S.F2_NAMES if n not in S.OPTIONAL_F2}
    pd = dict(S.DEFAULT_PD, dtm=dt / M, dt=dt)
    pi = {n: 0 for n in S.PI_NAMES}
    pi.update(M=M, MM=1, runtype=case.get("runtype", 4), vel2d_adv_split=HALFSPLIT, vel2d_adv_hor=P2_PDM,
              vel3d_adv_split=HALFSPLIT, vel3d_adv_hor=P2_PDM, vel3d_adv_ver=P2_PDM, temp_adv_split=HALFSPLIT,
              temp_adv_hor=P2_PDM, temp_adv_ver=P2_PDM, salt_adv_split=HALFSPLIT, salt_adv_hor=P2_PDM,
              salt_adv_ver=P2_PDM, adv_ver_iterations=1, ufirst2d=0, ufirst3d=1, calc_temp=1, calc_salt=1,
              ip_method=1, eqstate_method=case.get("eos", 1))
    md = pd["min_depth"]
    wet = az >= 1
    f2["H"] = H
    f2["HU"][:, :-1] = 0.5 * (H[:, :-1] + H[:, 1:])
    f2["HV"][:-1, :] = 0.5 * (H[:-1, :] + H[1:, :])
    cor = 2.0 * (2.0 * math.pi / 86164.0) * math.sin(math.radians(54.0))
    f2["coru"], f2["corv"] = cor * (au > 0).double(), cor * (av > 0).double()
    for n in ("zub0", "zvb0", "zub", "zvb"):
        f2[n].fill_(0.01)
    wind = _smooth(gen, g.nj, g.ni, g.ni / 6.0)
    f2["tausx"], f2["tausy"] = 0.05 + 0.02 * wind, 0.03 - 0.02 * wind
    f2["airp"] = 101300.0 + 200.0 * _smooth(gen, g.nj, g.ni, g.ni / 5.0)
    z = 0.05 * _smooth(gen, g.nj, g.ni, 4.0) * wet
    f2["z"], f2["zo"], f2["sseo"], f2["ssen"] = z.clone(), z.clone(), z.clone(), z.clone()
    f2["D"] = z + H
    f2["DU"][:, :-1] = (torch.maximum(0.5 * (z + _sh(z, 1, 0)), md - f2["HU"]) + f2["HU"])[:, :-1]
    f2["DV"][:-1, :] = (torch.maximum(0.5 * (z + _sh(z, 0, 1)), md - f2["HV"]) + f2["HV"])[:-1, :]
    for n, D, m, d0 in (("dry_z", "D", az, md), ("dry_u", "DU", au, 2 * md), ("dry_v", "DV", av, 2 * md)):
        f2[n] = torch.where(m > 0, torch.clamp((f2[D] - d0) / (pd["crit_depth"] - 2 * md), 0.0, 1.0), zero2())
    for old, new, D, h in (("ssuo", "ssun", "DU", "HU"), ("ssvo", "ssvn", "DV", "HV")):
        f2[old], f2[new] = f2[D] - f2[h], f2[D] - f2[h]
    f2["Dn"], f2["Dun"], f2["Dvn"] = f2["D"].clone(), f2["DU"].clone(), f2["DV"].clone()
    f2["U"], f2["V"] = _flow(gen, g, H, au, av)
    f2["Uinto"], f2["Vinto"] = f2["U"].clone(), f2["V"].clone()
    t = {"f2_" + n: a.contiguous() for n, a in f2.items()}
    t.update(az=az, au=au, av=av, ax=ax)
    # 3D fields: equidistant sigma layers, sheared velocities, stratified water, parabolic viscosity
    d3 = DTYPES[case["dtype"]]
    lev = torch.arange(kmax + 1, device=device, dtype=torch.float64)
    col = lambda a: (a[None] + 0 * lev[:, None, None]).to(d3).contiguous()  # noqa: E731
    for n, a in (("ho", f2["D"]), ("hn", f2["D"]), ("huo", f2["DU"]), ("hun", f2["DU"]), ("hvo", f2["DV"]), ("hvn", f2["DV"])):
        t["f3_" + n] = col(a / kmax)
    depth = 1.0 - (lev - 0.5) / kmax
    layer = (1.0 + 0.6 * (0.5 - depth)) * (lev > 0)
    for n, a in (("uu", f2["U"]), ("vv", f2["V"])):
        t["f3_" + n] = (a[None] / kmax * layer[:, None, None]).to(d3).contiguous()
    zero3 = lambda: torch.zeros(g.shape3(), dtype=d3, device=device)  # noqa: E731
    for n in ("ww", "uuEx", "vvEx", "idpdx", "idpdy", "rho", "buoy"):
        t["f3_" + n] = zero3()
    front = _smooth(gen, g.nj, g.ni, g.ni / 16.0)
    T, Sa = zero3(), zero3()
    for k in range(1, kmax + 1):
        d = float(depth[k])
        T[k] = ((20.0 - 12.0 * d + 0.8 * front * (1 - d) + 0.1 * _randn(gen, g.nj, g.ni)) * wet).to(d3)
        Sa[k] = ((30.0 + 5.0 * d - 0.5 * front + 0.02 * _randn(gen, g.nj, g.ni)) * wet).to(d3)
    t["f3_T"], t["f3_S"] = T, Sa
    buoy_of = -pd["g"] / pd["rho_0"]
    for k in range(1, kmax + 1):
        anom = pd["dtr0"] * (T[k].double() - pd["T0"]) + pd["dsr0"] * (Sa[k].double() - pd["S0"])
        t["f3_rho"][k] = (pd["rho_0"] + anom).to(d3)
        t["f3_buoy"][k] = (buoy_of * anom).to(d3)
    s = lev / kmax
    nu = (4 * 1e-2 * s * (1 - s) + 1e-6)[:, None, None]
    t["f3_num"] = (nu + torch.zeros(g.shape3(), dtype=torch.float64, device=device)).to(d3)
    t["f3_nuh"] = t["f3_num"].clone()
    if d3 == torch.float32:
        t["f3_Tlo"] = torch.zeros(g.shape3(), dtype=torch.float16, device=device)
        t["f3_Slo"] = torch.zeros(g.shape3(), dtype=torch.float16, device=device)
    return g, t, pd, pi, bdy


def _tracer_inputs(case, seed, device="cuda"):
    """(grid, tensors, dt): a closed basin with a sheared flow, ww by continuity."""
    g = Grid(case["nx"], case["ny"], case["kmax"], 500.0, 500.0)
    kmax, dt = g.kmax, 120.0
    gen = _gen(device, seed)
    az, H = _bathymetry("islands" if case["land"] > 0 else "flat", gen, g, case["land"])
    au, av, ax = _masks(az)
    U, V = _flow(gen, g, H, au, av, umax=0.8)
    HU, HV = 0.5 * (H + _sh(H, 1, 0)), 0.5 * (H + _sh(H, 0, 1))
    d3 = DTYPES[case["dtype"]]
    lev = torch.arange(kmax + 1, device=device, dtype=torch.float64)
    depth = 1.0 - (lev - 0.5) / kmax
    layer = ((1.0 + 0.8 * (0.5 - depth)) * (lev > 0))[:, None, None]
    on = (lev > 0).double()[:, None, None]
    t = dict(az=az, au=au, av=av, ax=ax)
    for n, a in (("ho", H), ("hn", H), ("hun", HU), ("hvn", HV)):
        t[n] = (torch.clamp(a, min=1.0)[None] / kmax * on).to(d3).contiguous()
    t["uu"], t["vv"] = ((a[None] / kmax * layer).to(d3).contiguous() for a in (U, V))
    ww = torch.zeros(g.shape3(), dtype=d3, device=device)
    w = torch.zeros(g.shape2(), dtype=torch.float64, device=device)
    for k in range(1, kmax):
        u, v = t["uu"][k].double(), t["vv"][k].double()
        w = w - ((u - _sh(u, -1, 0)) / g.dx + (v - _sh(v, 0, -1)) / g.dy)
        ww[k] = (w * (az == 1)).to(d3)
    t["ww"] = ww
    blob = _smooth(gen, g.nj, g.ni, max(2.0, g.ni / 24.0))
    f = torch.zeros(g.shape3(), dtype=d3, device=device)
    for k in range(1, kmax + 1):
        f[k] = ((10.0 + 2.0 * blob * (1.2 - float(depth[k])) + 0.05 * _randn(gen, g.nj, g.ni)) * (az >= 1)).to(d3)
    t["f"] = f
    s = lev / kmax
    t["nuh"] = ((4 * 5e-3 * s * (1 - s) + 1e-6)[:, None, None] * (1.0 + 0.3 * torch.tanh(blob))[None]).to(d3).contiguous()
    return g, t, dt


_TR = ("uu", "vv", "ww", "hun", "hvn", "ho", "hn", "nuh")


def _columns(case, seed, device="cuda"):
    """Coefficients au, bu, cu, du of diagonally dominant columns, laid out [level][column]."""
    gen = _gen(device, seed)
    shape = (case["kmax"] + 1, case["ncol"])
    au, cu = (-torch.rand(shape, generator=gen, device=device, dtype=torch.float64) for _ in range(2))
    return au, 1.0 - au - cu, cu, _randn(gen, *shape)


def prepare(case, seed):
    fam = case["family"]
    if fam == "tridiagonal":
        coef = _columns(case, seed)
        return dict(case=case, ctx=Context(Grid(8, 8, case["kmax"], 1.0, 1.0)), coef=coef,
                    value=torch.zeros_like(coef[1]))
    if fam in ("step", "density"):
        g, t, pd, pi, bdy = _state(case, seed)
        ctx = Context(g)
        st = BcDevice(tensors=t, pd=pd, pi=pi)
        ctx.init_advection(*st.masks())
        if bdy is not None:
            ctx.set_open_boundaries(bdy)
        return dict(case=case, ctx=ctx, st=st, n=1)
    g, t, dt = _tracer_inputs(case, seed)
    ctx = Context(g)
    ctx.init_advection(t["az"], t["au"], t["av"], t["ax"])
    s = dict(case=case, ctx=ctx, t=t, dt=dt)
    if fam == "gradient":
        s.update(f=torch.empty_like(t["f"]), weight=_weight(g, t), fbar=torch.empty_like(t["f"]),
                 nubar=torch.empty_like(t["f"]))
    return s


def _weight(g, t):
    """dJ/df of the tracer content of the basin's central quarter."""
    w = torch.zeros_like(t["f"])
    sl = (slice(1, None), slice(2 + g.ny // 4, 2 + 3 * g.ny // 4), slice(2 + g.nx // 4, 2 + 3 * g.nx // 4))
    w[sl] = t["hn"][sl] * (t["az"][sl[1:]] == 1)
    return w


# fields of a state that a step only reads
_READ_ONLY = ("f2_fwf", "f2_H", "f2_HU", "f2_HV", "f2_coru", "f2_corv", "f2_tausx", "f2_tausy", "f2_airp", "f2_zub0",
              "f2_zvb0", "f3_num", "f3_nuh")
# fields that the barotropic model (runtype 1) writes
_BAROTROPIC = ("z", "zo", "U", "V", "D", "DU", "DV", "UEx", "VEx", "fU", "fV", "ru", "rv", "ruu", "rvv", "zub", "zvb",
               "dry_z", "dry_u", "dry_v")


def _written(case, t):
    if case["family"] == "density":
        return ["f3_rho", "f3_buoy", "f3_idpdx", "f3_idpdy"]
    if case["runtype"] == 1:
        return ["f2_" + n for n in _BAROTROPIC]
    return [n for n in t if n[:3] in ("f2_", "f3_") and n not in _READ_ONLY + ("f2_zub", "f2_zvb")]


def run(state):
    case, ctx = state["case"], state["ctx"]
    fam = case["family"]
    if fam == "tridiagonal":
        ctx.tridiagonal(case["kmax"], 0, case["kmax"], *state["coef"], state["value"])
        return state["value"]
    if fam == "step":
        st = state["st"]
        ctx.time_loop(st, state["n"], case["M"])
        state["n"] += case["M"]
        return {n: st.t[n] for n in _written(case, st.t)}
    if fam == "density":
        st = state["st"]
        ctx.do_eqstate(st)
        ctx.internal_pressure(st)
        return {n: st.t[n] for n in _written(case, st.t)}
    t, dt, sch = state["t"], state["dt"], case["scheme"]
    if fam == "tracer":
        ctx.tracer_step(dt, t["f"], *[t[n] for n in _TR], HALFSPLIT, sch, sch, case["AH"], 0.9, 1.1e-9)
        return t["f"]
    state["f"].copy_(t["f"])
    state["fbar"].copy_(state["weight"])
    state["nubar"].zero_()
    ctx.tracer_gradient(case["nsteps"], case["every"], dt, state["f"], *[t[n] for n in _TR], HALFSPLIT, sch, sch,
                        case["AH"], 0.9, 1.1e-9, state["fbar"], state["nubar"])
    return {"f": state["f"], "fbar": state["fbar"], "nubar": state["nubar"]}


# --------------------------------------------------------------------------------------------------
# the same paths in plain 64-bit torch
F32 = S.F32
CNPAR, AVMOL = 0.9, 1.1e-9


def _div(a, b):
    """a / b, 0 where b is 0 (points outside the masks)."""
    ok = b != 0
    return torch.where(ok, a / torch.where(ok, b, torch.ones_like(b)), torch.zeros_like(a))


def _face_value(scheme, cfl, fuu, fu, fd):
    """Interface value of the limited schemes (adv_interfacial_reconstruction)."""
    df, du = fd - fu, fu - fuu
    x = (1.0 - 2.0 * cfl) / 6.0
    if scheme == P2:
        return fu + 0.5 * (1.0 - cfl) * ((0.5 + x) * df + (0.5 - x) * du)
    if scheme == UPSTREAM:
        return fu
    ok = df * du > 0
    r = torch.where(ok, du, torch.ones_like(du)) / torch.where(ok, df, torch.ones_like(df))
    two = 2.0 * torch.ones_like(r)
    if scheme == SUPERBEE:
        lim = torch.maximum(torch.minimum(2 * r, 0.5 * two), torch.minimum(r, two))
    elif scheme == MUSCL:
        lim = torch.minimum(torch.minimum(2 * r, 0.5 * (1 + r)), two)
    else:
        lim = torch.minimum(torch.minimum(2 * r / (cfl + 1e-10), (0.5 + x) + (0.5 - x) * r), 2.0 / (1.0 - cfl))
    return torch.where(ok, fu + 0.5 * lim * (1.0 - cfl) * df, fu)


def _sweep(axis, f, fi, D, U, DU, mflux, mupd, dt, frac, g, scheme, AH=0.0):
    """One split sweep along i (axis 0) or j (axis 1): (new f, new heights, flux divergence)."""
    s = (lambda a, q: _sh(a, q, 0)) if axis == 0 else (lambda a, q: _sh(a, 0, q))
    n = f.shape[-1] if axis == 0 else f.shape[-2]
    q = torch.arange(n, device=f.device)
    q = q[None, :] if axis == 0 else q[:, None]
    sub = 0 if scheme == UPSTREAM else 1
    dxf, dyf = (g.dx, g.dy) if axis == 0 else (g.dy, g.dx)
    dti = frac * dt
    on = mflux & (q >= sub) & (q <= n - 2 - sub)
    pos = U > 0
    fm, f1, f2 = s(f, -1), s(f, 1), s(f, 2)
    fu = torch.where(pos, f, f1)
    cfl = _div(U.abs(), DU) * (dti / dxf)
    val = _face_value(scheme, cfl, torch.where(pos, fm, f2), fu, torch.where(pos, f1, f))
    val = torch.where(torch.where(pos, s(mflux, -1), s(mflux, 1)), val, fu)
    flux = U * val
    if AH > 0:
        flux = flux - AH * DU * (f1 - f) / dxf
    flux = torch.where(on, flux, torch.zeros_like(flux))
    upd = mupd & (q >= 1 + sub) & (q <= n - 2 - sub)
    dD = dti * dyf * g.ard1 * (U - s(U, -1))
    adv = torch.where(upd, frac * dyf * g.ard1 * (flux - s(flux, -1)), torch.zeros_like(flux))
    Dn = torch.where(upd, D - dD, D)
    new = torch.where(upd, (D * fi - dt * adv) / torch.where(upd, Dn, torch.ones_like(Dn)), fi)
    return new, Dn, adv


def _sweep_w(f, h, ww, az, dt, scheme):
    """Vertical split sweep of all levels (level 0 first): (new f, new heights, flux divergence)."""
    on = (az == 1).clone()
    on[-1, :] = False
    on[:, -1] = False
    kmax = f.shape[0] - 1
    w = ww[1:kmax]
    fk, fk1 = f[1:kmax], f[2:kmax + 1]
    fkm = f[0:kmax - 1]
    fk2 = torch.cat((f[3:kmax + 1], torch.zeros_like(f[:1])), 0)
    pos = w > 0
    fu = torch.where(pos, fk, fk1)
    cfl = _div(w.abs() * dt, 0.5 * (h[1:kmax] + h[2:kmax + 1]))
    val = _face_value(scheme, cfl, torch.where(pos, fkm, fk2), fu, torch.where(pos, fk1, fk))
    k = torch.arange(1, kmax, device=f.device)[:, None, None]
    val = torch.where(torch.where(pos, k > 1, k < kmax - 1), val, fu)
    flux = torch.cat((torch.zeros_like(f[:1]), w * val, torch.zeros_like(f[:1])), 0)
    dh = dt * (ww[1:] - ww[:-1])
    adv = torch.where(on, flux[1:] - flux[:-1], torch.zeros_like(flux[1:]))
    hn = torch.where(on, h[1:] - dh, h[1:])
    new = torch.where(on, (h[1:] * f[1:] - dt * adv) / torch.where(on, hn, torch.ones_like(hn)), f[1:])
    return torch.cat((f[:1], new), 0), torch.cat((h[:1], hn), 0), adv


def _grid_masks(az, au, av, ax, grid):
    """Flux and update masks of the T, U and V advection grids (init_advection) and the grid's az."""
    H = az == 1
    uf, vf = (au == 1) | (au == 2), (av == 1) | (av == 2)
    uf, vf, xf = uf.clone(), vf.clone(), (ax == 1).clone()
    uf[:, -1] = False
    vf[-1, :] = False
    xf[:, -1] = False
    xf[-1, :] = False
    if grid == "H":
        return uf, vf, H, H, az
    if grid == "U":
        return _sh(H, 1, 0), xf, au == 1, uf, au
    return xf, _sh(H, 0, 1), vf, av == 1, av


def _advect(f, uu, vv, ww, hu, hv, ho, dt, g, m, scheme, AH=0.0, chunk=8):
    """do_advection_3d with HALFSPLIT (u/2 v/2 w v/2 u/2): (new f, summed flux divergence).
    The heights are functions level(k0, k1) so that large domains are widened a few levels at a
    time."""
    kmax = f.shape[0] - 1
    mfu, mfv, mpu, mpv, az = m
    one, two, H = f, [], []
    adv = []
    for a in range(1, kmax + 1, chunk):
        b = min(kmax + 1, a + chunk)
        x, D, a1 = _sweep(0, f[a:b], f[a:b], ho(a, b), uu(a, b), hu(a, b), mfu, mpu, dt, 0.5, g, scheme, AH)
        x, D, a2 = _sweep(1, x, x, D, vv(a, b), hv(a, b), mfv, mpv, dt, 0.5, g, scheme, AH)
        two.append(x)
        H.append(D)
        adv.append(a1 + a2)
    x, D, adv = torch.cat([one[:1]] + two, 0), torch.cat([torch.zeros_like(H[0][:1])] + H, 0), torch.cat(adv, 0)
    del two, H
    if kmax > 1:
        rows, parts = max(1, (1 << 26) // (x.shape[0] * x.shape[2])), []
        w = ww(0, kmax + 1)
        edge = torch.zeros_like(az, dtype=torch.bool)
        edge[:-1, :-1] = True
        azw = torch.where(edge, az, torch.zeros_like(az))
        for r in range(0, x.shape[1], rows):
            sl = (slice(None), slice(r, r + rows))
            pad = torch.nn.functional.pad(azw[sl[1]], (0, 1, 0, 1))  # _sweep_w leaves its last row and column
            wide = [torch.nn.functional.pad(q[sl], (0, 1, 0, 1)) for q in (x, D, w)]
            parts.append([q[:, :-1, :-1] for q in _sweep_w(wide[0], wide[1], wide[2], pad, dt, scheme)])
        x, D, aw = (torch.cat([p[q] for p in parts], 1) for q in range(3))
        adv = adv + aw
        del parts, aw, w
    out = [x[:1]]
    total = []
    for a in range(1, kmax + 1, chunk):
        b = min(kmax + 1, a + chunk)
        y, Dy, a4 = _sweep(1, x[a:b], x[a:b], D[a:b], vv(a, b), hv(a, b), mfv, mpv, dt, 0.5, g, scheme, AH)
        y, Dy, a5 = _sweep(0, y, y, Dy, uu(a, b), hu(a, b), mfu, mpu, dt, 0.5, g, scheme, AH)
        out.append(y)
        total.append(adv[a - 1:b - 1] + a4 + a5)
    return torch.cat(out, 0), torch.cat(total, 0)


def _vdiff(f, hn, nuh, az, dt, cnpar, avmol):
    """Implicit vertical diffusion of the interior water columns (salinity.F90:348-389)."""
    kmax = f.shape[0] - 1
    if kmax <= 1:
        return f
    on = torch.zeros_like(az, dtype=torch.bool)
    on[2:-2, 2:-2] = az[2:-2, 2:-2] == 1
    h = [None] + [torch.where(on, hn(k, k + 1)[0], torch.ones_like(hn(k, k + 1)[0])) for k in range(1, kmax + 1)]
    q = [None] + [2.0 * dt * (nuh(k, k + 1)[0] + avmol) / (h[k] + h[k + 1]) for k in range(1, kmax)] + [None]
    ru, qu = [None] * (kmax + 1), [None] * (kmax + 1)
    for k in range(kmax, 0, -1):
        up = q[k] if k < kmax else 0.0
        dn = q[k - 1] if k > 1 else 0.0
        rhs = f[k] * h[k]
        if k < kmax:
            rhs = rhs + (1 - cnpar) * up * (f[k + 1] - f[k])
        if k > 1:
            rhs = rhs - (1 - cnpar) * dn * (f[k] - f[k - 1])
        den = h[k] + cnpar * (up + dn)
        if k < kmax:
            den = den + cnpar * up * ru[k + 1]
            rhs = rhs + cnpar * up * qu[k + 1]
        ru[k] = -cnpar * dn / den if k > 1 else None
        qu[k] = rhs / den
    new = [None, qu[1]]
    for k in range(2, kmax + 1):
        new.append(qu[k] - ru[k] * new[k - 1])
    return torch.stack([f[0]] + [torch.where(on, new[k], f[k]) for k in range(1, kmax + 1)], 0)


def _levels(a):
    return lambda k0, k1: a[k0:k1].double()


def _plane(a):
    return lambda k0, k1: a[None].expand(k1 - k0, *a.shape)


def _tracer_step64(t, f, nuh, dt, g, scheme, AH):
    m = _grid_masks(t["az"], t["au"], t["av"], t["ax"], "H")
    f, _ = _advect(f, _levels(t["uu"]), _levels(t["vv"]), _levels(t["ww"]), _levels(t["hun"]), _levels(t["hvn"]),
                   _levels(t["ho"]), dt, g, m, scheme, AH)
    return _vdiff(f, _levels(t["hn"]), _levels(nuh), t["az"], dt, CNPAR, AVMOL)


def _advect_2d(U, V, DU, DV, t, g, dtm, grid, scheme):
    """uv_advect: the advection term of one depth-averaged momentum component (HALFSPLIT)."""
    s = (lambda a: _sh(a, 1, 0)) if grid == "U" else (lambda a: _sh(a, 0, 1))
    on = torch.ones_like(U)
    if grid == "U":
        on[:, -1] = 0
    else:
        on[-1, :] = 0
    X, DX = (U, DU) if grid == "U" else (V, DV)
    mfu, mfv, mpu, mpv, _ = _grid_masks(t["az"], t["au"], t["av"], t["ax"], grid)
    f = _div(X, DX) * on
    ua, va, dua, dva = (0.5 * (a + s(a)) * on for a in (U, V, DU, DV))
    f, D, a1 = _sweep(0, f, f, DX, ua, dua, mfu, mpu, dtm, 0.5, g, scheme)
    f, D, a2 = _sweep(1, f, f, D, va, dva, mfv, mpv, dtm, 1.0, g, scheme)
    _, _, a3 = _sweep(0, f, f, D, ua, dua, mfu, mpu, dtm, 0.5, g, scheme)
    return a1 + a2 + a3


def _where_(t, name, cond, value):
    t[name] = torch.where(cond, value, t[name])


def _micro(t, g, pd, pi, bdy, loop, ufirst):
    """integrate_2d on the 64-bit tensors t (keys without prefix); returns the next ufirst."""
    A = t
    az, au, av = A["az"], A["au"], A["av"]
    nj, ni = az.shape
    inner = torch.zeros_like(az, dtype=torch.bool)
    inner[2:-2, 2:-2] = True
    iu = torch.ones_like(inner)
    iu[:, -1] = False
    jv = torch.ones_like(inner)
    jv[-1, :] = False
    E, W, N_, S_ = (lambda a: _sh(a, 1, 0)), (lambda a: _sh(a, -1, 0)), (lambda a: _sh(a, 0, 1)), (lambda a: _sh(a, 0, -1))
    kappa, md, gr, rho, dtm, avm = pd["kappa"], pd["min_depth"], pd["g"], pd["rho_0"], pd["dtm"], pd["avmmol"]
    zero = torch.zeros_like(A["U"])
    # bottom friction
    qu, qv = _div(A["U"], A["DU"]), _div(A["V"], A["DV"])
    vl = torch.where(inner, 0.25 * (qv + E(qv) + S_(qv) + S_(E(qv))), zero)
    ul = torch.where(inner, 0.25 * (qu + W(qu) + N_(qu) + N_(W(qu))), torch.where(iu & (au > 0), qu, zero))
    for on, a, b, D, zb, zb0, rr, r in ((iu & (au > 0), qu, vl, "DU", "zub", "zub0", "ruu", "ru"),
                                        (jv & (av > 0), ul, qv, "DV", "zvb", "zvb0", "rvv", "rv")):
        HH = torch.clamp(A[D], min=md)
        sp = a * a + b * b
        drag = (kappa / torch.log((A[zb] + 0.5 * HH) / A[zb])) ** 2
        if pi["runtype"] == 1:
            zn = torch.minimum(HH, A[zb0] + 0.1 * avm / torch.clamp(torch.sqrt(drag * sp), min=avm))
            _where_(A, zb, on, zn)
            drag = (kappa / torch.log((zn + 0.5 * HH) / zn)) ** 2
        _where_(A, rr, on, drag)
        _where_(A, r, on, drag * torch.sqrt(sp))
    for n, grid in (("UEx", "U"), ("VEx", "V")):
        A[n] = _advect_2d(A["U"], A["V"], A["DU"], A["DV"], A, g, dtm, grid, pi["vel2d_adv_hor"])

    def velocity(u):
        s = E if u else N_
        z, H, D = A["z"], A["H"], A["D"]
        mn = lambda a: torch.clamp(a, max=md)  # noqa: E731
        zp, zm = torch.maximum(s(z), -H + mn(s(D))), torch.maximum(z, -s(H) + mn(D))
        zx = (zp - zm + (s(A["airp"]) - A["airp"]) / (rho * gr)) / (g.dx if u else g.dy)
        ts = A["tausx" if u else "tausy"]
        X, DX, sl = A["U" if u else "V"], A["DU" if u else "DV"], A["Slru" if u else "Slrv"]
        Slr = torch.where(X > 0, torch.clamp(sl, min=0.0), torch.clamp(sl, max=0.0))
        cor = -A["fV"] if u else A["fU"]
        rest = -0.5 * (ts + s(ts)) / rho + cor + A["UEx" if u else "VEx"] + A["SlUx" if u else "SlVx"] + Slr
        m = au if u else av
        on = inner & ((m == 1) | (m == 2))
        new = (X - dtm * (gr * DX * zx + A["dry_u" if u else "dry_v"] * rest)) / (1.0 + dtm * _div(A["ru" if u else "rv"], DX))
        _where_(A, "U" if u else "V", on, new)
        if not u and bdy is not None:  # mirror_bdy_2d on the western side: V points between open points
            col = g.imin - (g.imin - 2)
            A["V"][:, col] = torch.where(av[:, col] == 3, A["V"][:, col + 1], A["V"][:, col])
        if u:
            U = A["U"]
            c = A["corv"] * 0.25 * (W(U) + U + N_(W(U)) + N_(U))
            _where_(A, "fU", inner, torch.where(av >= 1, c, zero))
        else:
            V = A["V"]
            c = A["coru"] * 0.25 * (S_(V) + S_(E(V)) + V + E(V))
            _where_(A, "fV", inner, torch.where(au >= 1, c, zero))

    for u in ((True, False) if ufirst else (False, True)):
        velocity(u)
    if bdy is not None:
        fac = min(1.0, 4.0 * loop / bdy.ramp) if bdy.ramp > 1 else 1.0
        zb = float(bdy.amp[0]) * math.sin(2.0 * math.pi * (loop * dtm) / bdy.period + float(bdy.phase[0]))
        rows = slice(2, 2 + g.ny)
        A["z"] = A["z"].clone()
        A["z"][rows, 2] = torch.clamp(md - A["H"][rows, 2], min=fac * zb)
    if pi["runtype"] > 1:
        A["Uint"], A["Vint"] = A["Uint"] + A["U"], A["Vint"] + A["V"]
    A["zo"] = A["z"]
    div = ((A["U"] - W(A["U"])) * g.dy + (A["V"] - S_(A["V"])) * g.dx) * g.ard1
    _where_(A, "z", inner & (az == 1), A["z"] - dtm * div + dtm * A["fwf"])
    z, zo = A["z"], A["zo"]
    A["D"] = z + A["H"]
    d2 = pd["crit_depth"] - 2 * md
    for D, h, s, on in (("DU", "HU", E, iu), ("DV", "HV", N_, jv)):
        _where_(A, D, on, torch.maximum(0.25 * (zo + s(zo) + z + s(z)), md - A[h]) + A[h])
    for n, D, m, d0 in (("dry_z", "D", az, md), ("dry_u", "DU", au, 2 * md), ("dry_v", "DV", av, 2 * md)):
        _where_(A, n, m > 0, torch.clamp((A[D] - d0) / d2, 0.0, 1.0))
    return 0 if ufirst else 1


def _pressure(A, g, inner):
    """Blumberg-Mellor internal pressure: (idpdx, idpdy), rows of levels 0..kmax."""
    kmax = g.kmax
    out = []
    for h, m, s, d, old in (("hun", A["au"], lambda a: _sh(a, 1, 0), g.dx, "idpdx"),
                            ("hvn", A["av"], lambda a: _sh(a, 0, 1), g.dy, "idpdy")):
        on = inner & (m >= 1)
        hc = A["hn"][kmax].double()
        hx = A[h][kmax].double()
        res = A[old].double()
        res[0] = 0.0
        grdl = prgr = bl = None
        for k in range(kmax, 0, -1):
            b = A["buoy"][k].double()
            grad = (s(b) - b) / d
            mean = 0.5 * (s(b) + b)
            if k == kmax:
                prgr = grad * 0.5 * hx
            else:
                zz = k * hc - A["H"]
                prgr = prgr + 0.5 * (grdl + grad) * hx - (s(zz) - zz) / d * (bl - mean)
            grdl, bl = grad, mean
            res[k] = torch.where(on, hx * prgr, res[k])
        out.append(res)
    return out


def _unesco(T, Sa):
    c = F32
    T2, T3, T4, T5 = T * T, T ** 3, T ** 4, T ** 5
    x = c(999.842594) + c(6.793952e-02) * T - c(9.09529e-03) * T2 + c(1.001685e-04) * T3
    x = x - c(1.120083e-06) * T4 + c(6.536332e-09) * T5
    x = x + Sa * (c(0.824493) - c(4.0899e-03) * T + c(7.6438e-05) * T2 - c(8.2467e-07) * T3)
    x = x + Sa * c(5.3875e-09) * T4
    x = x + torch.sqrt(Sa ** 3) * (-c(5.72466e-03) + c(1.0227e-04) * T - c(1.6546e-06) * T2)
    return x + c(4.8314e-04) * Sa * Sa


def _density(A, pd, pi):
    """do_eqstate: rho and buoy of levels 1..kmax, in place."""
    x = -pd["g"] / pd["rho_0"]
    for k in range(1, A["T"].shape[0]):
        T, Sa = A["T"][k].double(), A["S"][k].double()
        if pi["eqstate_method"] == 1:
            rho = pd["rho_0"] + pd["dtr0"] * (T - pd["T0"]) + pd["dsr0"] * (Sa - pd["S0"])
        else:
            rho = torch.where(A["az"] > 0, _unesco(T, Sa), A["rho"][k].double())
        A["rho"][k] = rho
        A["buoy"][k] = x * (rho - pd["rho_0"])


def _macro(A, g, pd, pi):
    """integrate_3d on the 64-bit tensors A (3D fields FP64)."""
    kmax, dt, md = g.kmax, pd["dt"], pd["min_depth"]
    az, au, av = A["az"], A["au"], A["av"]
    shelf = bool((az == 2).any())
    inner = torch.zeros_like(az, dtype=torch.bool)
    inner[2:-2, 2:-2] = True
    iu = torch.ones_like(inner)
    iu[:, -1] = False
    jv = torch.ones_like(inner)
    jv[-1, :] = False
    E, W, N_, S_ = (lambda a: _sh(a, 1, 0)), (lambda a: _sh(a, -1, 0)), (lambda a: _sh(a, 0, 1)), (lambda a: _sh(a, 0, -1))
    # start_macro
    A["sseo"], A["ssen"] = A["ssen"], A["z"].clone()
    A["Dn"] = A["ssen"] + A["H"]
    for on, old, new, s, h, D in ((iu, "ssuo", "ssun", E, "HU", "Dun"), (jv, "ssvo", "ssvn", N_, "HV", "Dvn")):
        v = torch.maximum(0.25 * (A["sseo"] + s(A["sseo"]) + A["ssen"] + s(A["ssen"])), md - A[h])
        _where_(A, old, on, A[new])
        _where_(A, new, on, v)
        _where_(A, D, on, v + A[h])
    A["Uint"], A["Vint"] = A["Uint"] / pi["M"], A["Vint"] / pi["M"]
    # bottom_friction_3d
    qu, qv = _div(A["uu"][1], A["huo"][1]), _div(A["vv"][1], A["hvo"][1])
    for on, a, b, h, zb, r in (
            (inner & (au >= 1), qu, 0.25 * (qv + E(qv) + S_(qv) + S_(E(qv))), "hun", "zub", "rru"),
            (inner & (av >= 1), 0.25 * (qu + W(qu) + N_(qu) + N_(W(qu))), qv, "hvn", "zvb", "rrv")):
        hh = torch.clamp(A[h][1], min=md / kmax)
        x = pd["kappa"] / torch.log((A[zb] + 0.5 * hh) / A[zb])
        _where_(A, r, on, x * x * torch.sqrt(a * a + b * b))
    A["idpdx"], A["idpdy"] = _pressure(A, g, inner)

    def momentum(u):
        s = E if u else N_
        m = au if u else av
        on = inner & ((m == 1) | (m == 2))
        X, Y, h = A["uu" if u else "vv"], A["vv" if u else "uu"], A["hun" if u else "hvn"][kmax]
        hc = torch.where(on, h, torch.ones_like(h))
        dry, ts = A["dry_u" if u else "dry_v"], A["tausx" if u else "tausy"]
        cor = A["coru"] if u else -A["corv"]
        Ex, ip, r = A["uuEx" if u else "vvEx"], A["idpdx" if u else "idpdy"], A["rru" if u else "rrv"]
        H, D, so = A["H"], A["D"], A["sseo"]
        zp, zm = torch.maximum(s(so), -H + torch.clamp(s(D), max=md)), torch.maximum(so, -s(H) + torch.clamp(D, max=md))
        zx = (zp - zm + (s(A["airp"]) - A["airp"]) / (pd["g"] * pd["rho_0"])) / (g.dx if u else g.dy)
        ru, qu_ = [None] * (kmax + 1), [None] * (kmax + 1)
        q = [None] * (kmax + 1)
        for k in range(1, kmax):
            q[k] = 2.0 * dt * (0.5 * (A["num"][k] + s(A["num"][k])) + pd["avmmol"]) / (2.0 * hc)
        cn = pd["cnpar"]
        for k in range(kmax, 0, -1):
            y = Y[k]
            loc = 0.25 * (y + E(y) + S_(y) + S_(E(y))) if u else 0.25 * (y + W(y) + N_(y) + N_(W(y)))
            ex = dry * (cor * loc - Ex[k] + pd["ip_fac"] * ip[k])
            if k == kmax:
                ex = ex + dry * 0.5 * (ts + s(ts)) / pd["rho_0"]
            rhs = X[k] + dt * ex - dt * hc * pd["g"] * zx
            den = torch.ones_like(hc)
            if k < kmax:
                rhs = rhs + (1 - cn) * q[k] * (X[k + 1] - X[k]) / hc
                den = den + cn * q[k] / hc * (1.0 + ru[k + 1])
                rhs = rhs + cn * q[k] / hc * qu_[k + 1]
            if k > 1:
                rhs = rhs - (1 - cn) * q[k - 1] * (X[k] - X[k - 1]) / hc
                den = den + cn * q[k - 1] / hc
            else:
                den = den + dt * r / hc
            qu_[k] = rhs / den
            ru[k] = -cn * q[k - 1] / hc / den if k > 1 else None
        v, total = [None, qu_[1]], qu_[1]
        for k in range(2, kmax + 1):
            v.append(qu_[k] - ru[k] * v[k - 1])
            total = total + v[k]
        ss, HX, I = A["ssuo" if u else "ssvo"], A["HU" if u else "HV"], A["Uint" if u else "Vint"]
        diff = (I - total) / torch.where(on, ss + HX, torch.ones_like(ss))
        for k in range(1, kmax + 1):
            X[k] = torch.where(on, v[k] + h * diff, X[k])
        if shelf and not u:  # mirror_bdy_3d on the western side
            X[:, :, 2] = torch.where(av[None, :, 2] == 3, X[:, :, 3], X[:, :, 2])

    for u in ((True, False) if pi["ufirst3d"] else (False, True)):
        momentum(u)
    # sigma_coordinates
    for n, e, h, on in (("ho", "sseo", "H", None), ("hn", "ssen", "H", None), ("huo", "ssuo", "HU", iu),
                        ("hun", "ssun", "HU", iu), ("hvo", "ssvo", "HV", jv), ("hvn", "ssvn", "HV", jv)):
        v = ((A[e] + A[h]) / kmax)[None].expand(kmax + 1, *az.shape)
        A[n] = v.clone() if on is None else torch.where(on, v, A[n])
    # ww_momentum_3d
    w, rate = A["ww"][0].clone(), (A["hn"][1] - A["ho"][1]) / dt
    for k in range(1, kmax):
        u, v = A["uu"][k], A["vv"][k]
        w = w - rate - ((u - W(u)) * g.dy + (v - S_(v)) * g.dx) * g.ard1
        A["ww"][k] = torch.where(inner & (az == 1), w, A["ww"][k])
    # uv_advect_3d
    for n, x, grid, s, on in (("uuEx", "uu", "U", E, iu), ("vvEx", "vv", "V", N_, jv)):
        h2 = A["hun" if grid == "U" else "hvn"][1]
        f = torch.where(on, _div(A[x], h2[None].expand_as(A[x])), torch.zeros_like(A[x]))
        f[0] = 0.0
        mean = lambda a: lambda k0, k1: torch.where(on, 0.5 * (a[k0:k1] + s(a[k0:k1])), torch.zeros_like(a[k0:k1]))  # noqa: E731
        both = torch.where(on, 0.5 * (s(A["ho"][1]) + s(A["hn"][1])), torch.zeros_like(h2))
        other = A["hvn" if grid == "U" else "hun"][1]
        other = torch.where(on & iu & jv, 0.5 * (other + s(other)), torch.zeros_like(h2))
        hu, hv = (both, other) if grid == "U" else (other, both)
        wa = mean(A["ww"])
        wsurf = lambda k0, k1: wa(k0, k1) * (torch.arange(k0, k1, device=f.device) > 0)[:, None, None]  # noqa: E731
        m = _grid_masks(az, au, av, A["ax"], grid)
        _, adv = _advect(f, mean(A["uu"]), mean(A["vv"]), wsurf, _plane(hu), _plane(hv), _plane(h2), dt, g, m,
                         pi["vel3d_adv_hor"])
        A[n] = torch.cat((torch.zeros_like(adv[:1]), adv), 0)
        del f, adv
    # stresses_3d
    tx, ty = -_div(A["uu"][1], A["hun"][1]) * A["rru"], -_div(A["vv"][1], A["hvn"][1]) * A["rrv"]
    rowi, coli = torch.zeros_like(inner), torch.zeros_like(inner)
    rowi[2:-2, 1:-2] = True
    coli[1:-2, 2:-2] = True
    _where_(A, "taubx", rowi, tx)
    _where_(A, "tauby", coli, ty)
    _where_(A, "taub", inner, torch.sqrt(0.5 * (W(tx) ** 2 + tx ** 2 + S_(ty) ** 2 + ty ** 2)))
    _where_(A, "taus", inner, torch.sqrt(A["tausx"] ** 2 + A["tausy"] ** 2) / pd["rho_0"])
    # temperature and salinity
    m = _grid_masks(az, au, av, A["ax"], "H")
    for n, mol in (("T", "avmolt"), ("S", "avmols")):
        f, _ = _advect(A[n], _levels(A["uu"]), _levels(A["vv"]), _levels(A["ww"]), _plane(A["hun"][1]),
                       _plane(A["hvn"][1]), _plane(A["ho"][1]), dt, g, m, pi["temp_adv_hor"])
        f = _vdiff(f, _plane(A["hn"][1]), _levels(A["nuh"]), az, dt, pd["cnpar"], pd[mol])
        if shelf:
            f[:, :, 1] = torch.where(az[None, :, 2] > 1, f[:, :, 2], f[:, :, 1])
        A[n] = f
        del f
    _density(A, pd, pi)
    # slow_bottom_friction
    Ui, Vi = _div(A["Uinto"], A["ssuo"] + A["HU"]), _div(A["Vinto"], A["ssvo"] + A["HV"])
    ring_u, ring_v = torch.zeros_like(inner), torch.zeros_like(inner)
    ring_u[-2, :], ring_u[:, 1] = True, True
    ring_v[1, :], ring_v[:, -2] = True, True
    Ui = torch.where(inner & (au >= 1) | ~inner & ring_u, Ui, torch.zeros_like(Ui))
    Vi = torch.where(inner & (av >= 1) | ~inner & ring_v, Vi, torch.zeros_like(Vi))
    for m_, a, b, ss, h, zb, r in (
            (au, Ui, 0.25 * (Vi + E(Vi) + S_(Vi) + S_(E(Vi))), "ssun", "HU", "zub", "ru"),
            (av, 0.25 * (Ui + W(Ui) + N_(Ui) + N_(W(Ui))), Vi, "ssvn", "HV", "zvb", "rv")):
        hh = torch.clamp(A[ss] + A[h], min=md)
        x = pd["kappa"] / torch.log((A[zb] + 0.5 * hh) / A[zb])
        _where_(A, r, inner, torch.where(m_ >= 1, x * x * torch.sqrt(a * a + b * b), torch.zeros_like(a)))
    for n, grid in (("UEx", "U"), ("VEx", "V")):
        A[n] = _advect_2d(A["Uint"], A["Vint"], A["Dun"], A["Dvn"], A, g, pd["dtm"], grid, pi["vel2d_adv_hor"])
    # slow_terms
    for m_, Sl, Ex2, Ex3, ip, Slr, I, so, sn, h, r2, x, ho, hn, r3 in (
            (au, "SlUx", "UEx", "uuEx", "idpdx", "Slru", "Uint", "ssuo", "ssun", "HU", "ru", "uu", "huo", "hun", "rru"),
            (av, "SlVx", "VEx", "vvEx", "idpdy", "Slrv", "Vint", "ssvo", "ssvn", "HV", "rv", "vv", "hvo", "hvn", "rrv")):
        on = inner & (m_ >= 1)
        vs = -A[Ex2]
        for k in range(1, kmax + 1):
            vs = vs + A[Ex3][k] - pd["ip_fac"] * A[ip][k]
        _where_(A, Sl, on, vs)
        _where_(A, Slr, on, -_div(A[I], 0.5 * (A[so] + A[sn]) + A[h]) * A[r2] +
                _div(A[x][1], 0.5 * (A[ho][1] + A[hn][1])) * A[r3])
    A["Uinto"], A["Vinto"] = A["Uint"], A["Vint"]
    A["Uint"], A["Vint"] = torch.zeros_like(A["Uint"]), torch.zeros_like(A["Vint"])


def _step64(g, t, pd, pi, bdy, M):
    """The pass of a step case from the tensors of _state, in 64 bits."""
    A = {n[3:] if n[:3] in ("f2_", "f3_") else n: (a.double() if a.is_floating_point() else a) for n, a in t.items()
         if n not in ("f3_Tlo", "f3_Slo")}
    ufirst = pi["ufirst2d"]
    for n in range(1, M + 1):
        ufirst = _micro(A, g, pd, pi, bdy, n, ufirst)
    if pi["runtype"] > 1:
        _macro(A, g, pd, pi)
    return A


def exact(case, seed):
    fam = case["family"]
    if fam == "tridiagonal":
        au, bu, cu, du = _columns(case, seed)
        kmax = case["kmax"]
        ru, qu, v = [None] * (kmax + 1), [None] * (kmax + 1), torch.zeros_like(bu)
        for k in range(kmax, -1, -1):
            den = bu[k] if k == kmax else bu[k] - cu[k] * ru[k + 1]
            qu[k] = (du[k] if k == kmax else du[k] - cu[k] * qu[k + 1]) / den
            ru[k] = au[k] / den
        v[0] = qu[0]
        for k in range(1, kmax + 1):
            v[k] = qu[k] - ru[k] * v[k - 1]
        return v
    if fam == "step":
        g, t, pd, pi, bdy = _state(case, seed)
        A = _step64(g, t, pd, pi, bdy, case["M"])
        return {n: A.get(n[3:]) for n in _written(case, t)}
    if fam == "density":
        g, t, pd, pi, _ = _state(case, seed)
        A = {n[3:] if n[:3] in ("f2_", "f3_") else n: a for n, a in t.items()}
        A["rho"], A["buoy"] = A["rho"].double(), A["buoy"].double()
        _density(A, pd, pi)
        inner = torch.zeros_like(A["az"], dtype=torch.bool)
        inner[2:-2, 2:-2] = True
        ipx, ipy = _pressure(A, g, inner)
        return {"f3_rho": A["rho"], "f3_buoy": A["buoy"], "f3_idpdx": ipx, "f3_idpdy": ipy}
    g, t, dt = _tracer_inputs(case, seed)
    f = t["f"].double()
    if fam == "tracer":
        return _tracer_step64(t, f, t["nuh"], dt, g, case["scheme"], case["AH"])
    f0 = f.requires_grad_(True)
    nuh = t["nuh"].double().requires_grad_(True)
    f = f0
    for _ in range(case["nsteps"]):
        f = _tracer_step64(t, f, nuh, dt, g, case["scheme"], case["AH"])
    fbar, nubar = torch.autograd.grad(f, (f0, nuh), _weight(g, t).double())
    return {"f": f.detach(), "fbar": fbar, "nubar": nubar}
