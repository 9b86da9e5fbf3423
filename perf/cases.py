"""Workloads of the library, as a program that uses it runs them.

Every case is a dict of plain values.  `prepare` makes what the program has in
hand (seeded fields in pinned or ordinary host memory, a context with its
geometry, an ensemble, an adjoint), `run` does one job through the public
entry points and returns the fields it computed, `exact` restates the same
job in FP64 torch without the library.

The resident API keeps its fields on the GPU between calls and is fed from and
read back to host arrays, so a job is: upload the starting fields, compute,
download the results.  The Fortran drop-ins work on host arrays by their
nature.  `nse_spn_noalloc` works on the caller's device arrays.

Kinds (the sizes come from the repository's workloads, tests and benchmark):
  step      project a noisy penalised channel, then N time steps (FP64/mixed)
  ensemble  several small cases stepped together
  adjoint   gradient of the wall heat flux with respect to mask and state
  levelset  reinitialisation sweeps and the mask of a new geometry
  poisson   one pressure solve for a new right-hand side
  mkp       the projection drop-in on host arrays (a Fortran driver's call)
  spn       the spectral tridiagonal solve on device arrays

A padded field is (nx+2, ny+2, nz+2) with x fastest, held here as a C-ordered
(nz+2, ny+2, nx+2) tensor.
"""
import ctypes as C
import math

import numpy as np
import torch

from vtkmakecompare_b200 import lib
from vtkmakecompare_b200 import legacy
from vtkmakecompare_b200 import solver as S

XL, YL, ZL = 2 * math.pi, 2.0, math.pi
Y0, GAMMA = -1.0, 2.0
RE, PR, ETA = 3000.0, 0.71, 1.0e4
F64 = torch.float64


# ------------------------------------------------------------------- cases
def listed():
    return [
        # smallest channel of the benchmark, no obstacle: launches and latency
        dict(name="step64", kind="step", nx=64, ny=64, nz=64, steps=10, mixed=False,
             obstacle="none", t_bot=1.0),
        # a grid that is not a multiple of 32 in x: what a user's own mesh looks like
        dict(name="step_ragged", kind="step", nx=100, ny=75, nz=90, steps=20, mixed=False,
             obstacle="sphere", t_bot=0.0),
        # an ordinary case
        dict(name="step128", kind="step", nx=128, ny=96, nz=128, steps=50, mixed=False,
             obstacle="sphere", t_bot=0.0),
        # the headline workload: penalised channel with a sphere and heat
        dict(name="step256", kind="step", nx=256, ny=192, nz=256, steps=50, mixed=False,
             obstacle="sphere", t_bot=0.0),
        # the same in the mixed-precision form
        dict(name="mixed256", kind="step", nx=256, ny=192, nz=256, steps=50, mixed=True,
             obstacle="sphere", t_bot=0.0),
        # a batch of small cases (a parameter sweep) on eight streams
        dict(name="ensemble8", kind="ensemble", cases=8, steps=21, size=1.0),
        # shape optimisation: gradient over a checkpointed forward run
        dict(name="adjoint128", kind="adjoint", nx=128, ny=128, nz=128, steps=20, every=10,
             obstacle="sphere", t_bot=1.0),
        # a new geometry on an ordinary grid, the reference's 2000 sweeps
        dict(name="levelset128", kind="levelset", nx=128, ny=96, nz=128, sweeps=2000,
             obstacle="sphere"),
        # one pressure solve of the headline grid for a new right-hand side
        dict(name="poisson256", kind="poisson", nx=256, ny=192, nz=256),
        # a Fortran driver's projection on host arrays
        dict(name="mkp96", kind="mkp", nx=96, ny=64, nz=96, obstacle="none", t_bot=1.0),
        # the spectral solve for callers that own their device memory
        dict(name="spn128", kind="spn", nx=128, ny=96, nz=128),
    ]


def _smooth(lo, hi):
    """lengths the transforms take: products of 2, 3 and 5"""
    out = []
    for n in range(lo, hi + 1):
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            out.append(n)
    return out


def _near(values, x):
    return min(values, key=lambda v: abs(v - x))


def _grid(rng, lo, hi, regular=False):
    """nx, ny, nz around one size drawn on a logarithmic scale; x and z lengths
    have small prime factors, y is any number; `regular`: x as the mixed form
    needs it"""
    s = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    xs = [96, 128, 160, 192, 256] if regular else _smooth(24, 320)
    nx = _near(xs, s * rng.uniform(0.85, 1.2))
    nz = _near(_smooth(24, 320), s * rng.uniform(0.7, 1.1))
    ny = max(12, min(256, int(s * rng.uniform(0.5, 0.95))))
    return nx, ny, nz


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["mixed"] * 2 + ["ensemble", "adjoint", "levelset",
                                                       "levelset", "poisson", "mkp", "spn"])
    obstacle = rng.choice(["none", "sphere", "sphere", "boxes"])
    t_bot = rng.choice([0.0, 1.0])
    if kind in ("step", "mixed"):
        regular = kind == "mixed" or rng.random() < 0.5
        nx, ny, nz = _grid(rng, 40, 240, regular)
        steps = int(max(5, min(rng.uniform(8, 51), 5e8 / (nx * ny * nz))))
        return dict(kind="step", nx=nx, ny=ny, nz=nz, steps=steps, mixed=kind == "mixed",
                    obstacle=obstacle, t_bot=t_bot)
    if kind == "ensemble":
        return dict(kind="ensemble", cases=rng.randrange(3, 11), steps=rng.randrange(7, 30),
                    size=rng.choice([0.75, 1.0]))
    if kind == "adjoint":
        nx, ny, nz = _grid(rng, 40, 120, rng.random() < 0.5)
        return dict(kind="adjoint", nx=nx, ny=ny, nz=nz, steps=rng.randrange(6, 17),
                    every=rng.randrange(3, 9), obstacle="sphere", t_bot=1.0)
    if kind == "levelset":
        nx, ny, nz = _grid(rng, 40, 125)
        return dict(kind="levelset", nx=nx, ny=ny, nz=nz, sweeps=rng.choice([500, 1000, 2000]),
                    obstacle=rng.choice(["sphere", "boxes"]))
    if kind == "poisson":
        nx, ny, nz = _grid(rng, 40, 240)
        return dict(kind="poisson", nx=nx, ny=ny, nz=nz)
    if kind == "mkp":
        nx, ny, nz = _grid(rng, 32, 128)
        return dict(kind="mkp", nx=nx, ny=ny, nz=nz, obstacle="none", t_bot=t_bot)
    nx, ny, nz = _grid(rng, 32, 140)
    return dict(kind="spn", nx=nx, ny=ny, nz=nz)


# -------------------------------------------------------------------- work
def work(case):
    """bytes: what each pass of the job reads and writes once (FP64 unless the
    mixed form holds it in FP32), flops: FP64 operations of the transforms
    and stencils, rounded"""
    k = case["kind"]
    if k == "ensemble":
        n = sum(a * b * c for a, b, c, *_ in _ensemble_specs(case, 0))
        return {"bytes": (232.0 * case["steps"] + 72.0) * n, "flops": 700.0 * case["steps"] * n}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = float(nx * ny * nz)
    spec = 16.0 * (nx // 2 + 1) * ny * nz
    if k == "step":
        # per step: 25 field passes and four passes over the half spectrum;
        # per job: four fields in, five out
        s = 4.0 if case["mixed"] else 8.0
        per = (13 * 8.0 + 12 * s) * n + 4 * spec
        return {"bytes": per * case["steps"] + 9 * 8.0 * n, "flops": 700.0 * case["steps"] * n}
    if k == "adjoint":
        # a forward run, its replay, and a reverse step of twice a step's traffic
        per = 25 * 8.0 * n + 4 * spec
        return {"bytes": 4 * per * case["steps"] + 9 * 8.0 * n, "flops": 3000.0 * case["steps"] * n}
    if k == "levelset":
        # per sweep: the level set and the sign of phi0 in, the level set out
        return {"bytes": 24.0 * n * (case["sweeps"] + 1), "flops": 45.0 * n * (case["sweeps"] + 1)}
    if k == "poisson":
        return {"bytes": 16.0 * n + 4 * spec, "flops": 60.0 * n}
    if k == "mkp":
        # seven fields in (u_temp, p, u_ta), eleven out, the solve between
        return {"bytes": 18 * 8.0 * n + 4 * spec, "flops": 100.0 * n}
    return {"bytes": 2 * spec, "flops": 10.0 * spec / 16}


# ------------------------------------------------------------------ inputs
def grid(nx, ny, nz):
    """cell centres, faces and spacings of the channel mesh (x, z uniform, y
    with tanh-stretched faces), index 0..n+1"""
    g = {}
    for d, n, L in (("x", nx, XL), ("z", nz, ZL)):
        i = np.arange(n + 2, dtype=np.float64)
        f, c = L * i / n, L * (i - 0.5) / n
        d12 = np.empty(n + 2)
        d12[:-1] = c[1:] - c[:-1]
        d12[-1] = 2.0 * (f[-1] - c[-1])
        dd = np.empty(n + 2)
        dd[1:] = f[1:] - f[:-1]
        dd[0], dd[-1] = dd[1], dd[n]
        g[d], g[d + "12"], g["d" + d], g["d" + d + "12"] = c, f, dd, d12
    f = np.empty(ny + 2)
    for j in range(ny + 1):
        f[j] = Y0 + 0.5 * YL * (1.0 + math.tanh(GAMMA * (2.0 * j / ny - 1.0)) / math.tanh(GAMMA))
    f[ny + 1] = 2.0 * f[ny] - f[ny - 1]
    c = np.empty(ny + 2)
    c[1:ny + 1] = 0.5 * (f[:ny] + f[1:ny + 1])
    c[0], c[ny + 1] = 2.0 * f[0] - c[1], 2.0 * f[ny] - c[ny]
    d12 = np.empty(ny + 2)
    d12[:-1] = c[1:] - c[:-1]
    d12[-1] = 2.0 * (f[-1] - c[-1])
    dd = np.empty(ny + 2)
    dd[1:] = f[1:] - f[:-1]
    dd[0], dd[-1] = dd[1], dd[ny]
    g["y"], g["y12"], g["dy"], g["dy12"] = c, f, dd, d12
    return g


def _rand(shape, seed):
    gen = torch.Generator("cuda").manual_seed(int(seed))
    return torch.randn(shape, generator=gen, dtype=F64, device="cuda")


def _pad(x):
    out = torch.zeros([n + 2 for n in x.shape], dtype=F64, device=x.device)
    out[1:-1, 1:-1, 1:-1] = x
    return out


def _t(a):
    return torch.as_tensor(a, dtype=F64, device="cuda")


def obstacle_phi(g, kind, seed):
    """level set of the obstacle (positive inside), interior (nz, ny, nx): a
    sphere of the benchmark's radius, or one to three seeded spheres and boxes"""
    X, Y, Z = _t(g["x"][1:-1]), _t(g["y"][1:-1])[:, None], _t(g["z"][1:-1])[:, None, None]
    rng = np.random.default_rng(seed)

    def sphere(c, r):
        return r - torch.sqrt((X - c[0]) ** 2 + (Y - c[1]) ** 2 + (Z - c[2]) ** 2)

    if kind == "sphere":
        jit = rng.uniform(-0.05, 0.05, 3)
        return sphere((math.pi + jit[0], jit[1], math.pi / 2 + jit[2]), 0.25)
    phi = None
    for _ in range(int(rng.integers(1, 4))):
        r = float(rng.uniform(0.1, 0.3))
        c = (float(rng.uniform(0, XL)), float(rng.uniform(-0.9 + r, 0.9 - r)),
             float(rng.uniform(0, ZL)))
        if rng.random() < 0.5:
            p = sphere(c, r)
        else:
            q = torch.broadcast_tensors((X - c[0]).abs() - r, (Y - c[1]).abs() - r,
                                        (Z - c[2]).abs() - r)
            out = torch.sqrt(sum(a.clamp(min=0.0) ** 2 for a in q))
            p = -(out + torch.maximum(torch.maximum(q[0], q[1]), q[2]).clamp(max=0.0))
        phi = p if phi is None else torch.maximum(phi, p)
    return phi


def _smooth_mask(g, phi, width):
    h = width * _t(g["dx"][1:-1])
    c = (torch.sin(3.1415926535 * phi / 2.0 / h) + 1.0) / 2.0
    return torch.where(phi >= h, torch.ones_like(c), torch.where(phi <= -h, torch.zeros_like(c), c))


def channel(nx, ny, nz, seed, obstacle, t_bot, Re=RE):
    """seeded noisy channel: interior fields, mask, parameters"""
    g = grid(nx, ny, nz)
    ey = _t(g["y"][1:-1])[:, None]  # walls at -1 and 1
    noise = 0.05 * _rand((3, nz, ny, nx), seed)
    f = {"u": 1.5 * (1.0 - ey ** 2) + noise[0], "v": noise[1].clone(), "w": noise[2].clone(),
         "T": (t_bot * (1.0 - (ey + 1.0) / 2.0)).expand(nz, ny, nx).contiguous()}
    f["T"] = f["T"] + 0.01 * _rand((nz, ny, nx), seed + 7919)
    f["v"][:, -1] = 0.0
    c1 = torch.zeros((nz, ny, nx), dtype=F64, device="cuda")
    if obstacle != "none":
        c1 = _smooth_mask(g, obstacle_phi(g, obstacle, seed), 1.5)
    cfl = (f["u"].abs() / _t(g["dx"][1:-1]) + f["v"].abs() / _t(g["dy"][1:-1])[:, None] +
           f["w"].abs() / _t(g["dz"][1:-1])[:, None, None])
    # one fixed time step, three significant digits, at a Courant number of 0.4
    dt = float("%.2e" % (0.4 / float(cfl.max())))
    par = dict(dt=dt, Re=Re, Sc=PR, eta=ETA, force=3.0 / Re, source=0.0, tbot=t_bot, ttop=0.0,
               tsolid=1.0)
    return g, f, c1, par


def _pinned(x):
    p = torch.empty(x.shape, dtype=F64, pin_memory=True)
    p.copy_(x)
    return p


def _context(nx, ny, nz, par, c1, precision=S.FP64):
    cfg = S.Config(nx, ny, nz, par["dt"], par["Re"], par["Sc"], par["eta"], XL, YL, ZL, y0=Y0,
                   ystretch=GAMMA, body_force=par["force"], heat_source=par["source"],
                   t_bot=par["tbot"], t_top=par["ttop"], t_solid=par["tsolid"],
                   precision=precision)
    ctx = S.Context(cfg)
    ctx.upload_ptr("cellvalue", _pinned(c1).data_ptr())
    return ctx


def _ensemble_specs(case, seed):
    """grids, Reynolds numbers and seeds of an ensemble; the grids depend on the
    case alone (a sweep's plan), the fields and obstacles on the seed"""
    rng = np.random.default_rng(1000 * case["cases"] + case["steps"])
    grids = ((64, 64, 64), (96, 64, 96), (128, 96, 128), (160, 128, 160))
    out = []
    for i in range(case["cases"]):
        nx, ny, nz = grids[int(rng.integers(len(grids)))]
        if case["size"] != 1.0 and nx > 64:
            nx, ny, nz = (int(32 * round(case["size"] * n / 32)) for n in (nx, ny, nz))
        out.append((nx, ny, nz, float(rng.uniform(1000.0, 5000.0)), seed * 131 + i))
    return out


def _levelset_input(case, seed):
    """a level set whose slope varies around 1, as a geometry tool gives it"""
    g = grid(case["nx"], case["ny"], case["nz"])
    phi = obstacle_phi(g, case["obstacle"], seed)
    return g, phi * (1.0 + 0.3 * torch.sin(2.0 * _t(g["x"][1:-1])))


def _wrap_samples(x):
    """padded samples with the periodic fill of MKP: index 0 holds cell n"""
    f = _pad(x)
    f[0], f[:, :, 0] = f[-2], f[:, :, -2]
    f[0, :, 0] = f[-2, :, -2]
    return f


def _poisson_input(g, case, seed):
    """N(0,1) right-hand side without its dy-weighted mean"""
    r = _rand((case["nz"], case["ny"], case["nx"]), seed)
    dy = _t(g["dy"][1:-1])
    return r - (r.mean(dim=(0, 2)) * dy).sum() / dy.sum()


def _mkp_input(case, seed):
    """u_temp after SET_BC, and what MKP updates in place"""
    g, f, _, par = channel(case["nx"], case["ny"], case["nz"], seed, "none", case["t_bot"])
    us = {"us": bc_u(f["u"]), "vs": bc_v(f["v"]), "ws": bc_u(f["w"])}
    shape = us["us"].shape
    rest = {n: 1e-3 * _rand(shape, seed + 17 * i)
            for i, n in enumerate(("p", "u_ta", "v_ta", "w_ta"), 1)}
    return g, us, rest, par["dt"]


def _coeffs(g):
    """the y second difference (ny, 3) and the x-z symbols (nz+1, nx/2+1)"""
    nx, nz = len(g["x"]) - 2, len(g["z"]) - 2
    dy, dy12 = g["dy"][1:-1], g["dy12"]
    a, c = 1.0 / dy12[:-2] / dy, 1.0 / dy12[1:-1] / dy
    i, k = np.arange(nx // 2 + 1), np.arange(nz + 1)
    kx = i / XL * math.pi * 2.0
    kz = np.where(k <= nz // 2, k, k - nz) / ZL * math.pi * 2.0
    dx, dz = g["dx"][1], g["dz"][1]
    kxz = (2.0 * (1.0 - np.cos(kx * dx)) / dx / dx)[None, :] + \
          (2.0 * (1.0 - np.cos(kz * dz)) / dz / dz)[:, None]
    return _t(np.stack([a, -a - c, c], axis=1)), _t(kxz)


def _spn_input(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    AC, KXZ = _coeffs(grid(nx, ny, nz))
    return AC, KXZ.contiguous(), _rand((nz + 2, ny + 2, nx // 2 + 1, 2), seed)


# ------------------------------------------------------------ prepare / run
OUT = ("u", "v", "w", "p", "T")


def _buffers(shape, names):
    return {k: torch.empty(shape, dtype=F64, pin_memory=True) for k in names}


def prepare(case, seed):
    k = case["kind"]
    if k == "ensemble":
        st = dict(kind=k, steps=case["steps"], ctx=[], host=[], out=[])
        for nx, ny, nz, Re, s in _ensemble_specs(case, seed):
            _, f, c1, par = channel(nx, ny, nz, s, "boxes", 1.0, Re)
            st["ctx"].append(_context(nx, ny, nz, par, c1))
            st["host"].append({n: _pinned(_pad(x)) for n, x in f.items()})
            st["out"].append(_buffers((nz + 2, ny + 2, nx + 2), OUT))
        st["ens"] = S.Ensemble(st["ctx"], nstreams=8)
        return st
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    shape = (nz + 2, ny + 2, nx + 2)
    if k == "step":
        _, f, c1, par = channel(nx, ny, nz, seed, case["obstacle"], case["t_bot"])
        ctx = _context(nx, ny, nz, par, c1, S.MIXED if case["mixed"] else S.FP64)
        return dict(kind=k, steps=case["steps"], ctx=ctx,
                    host={n: _pinned(_pad(x)) for n, x in f.items()}, out=_buffers(shape, OUT))
    if k == "adjoint":
        _, f, c1, par = channel(nx, ny, nz, seed, case["obstacle"], case["t_bot"])
        ctx = _context(nx, ny, nz, par, c1)
        adj = S.Adjoint(ctx, case["steps"], checkpoint_every=case["every"],
                        avg_from=max(1, case["steps"] // 2))
        return dict(kind=k, ctx=ctx, adj=adj, host={n: _pinned(_pad(x)) for n, x in f.items()})
    if k == "levelset":
        g, phi0 = _levelset_input(case, seed)
        ctx = _context(nx, ny, nz, dict(dt=1e-3, Re=RE, Sc=PR, eta=ETA, force=0.0, source=0.0,
                                        tbot=0.0, ttop=0.0, tsolid=0.0), phi0 * 0.0)
        return dict(kind=k, ctx=ctx, sweeps=case["sweeps"],
                    phi0=_pad(phi0).cpu().numpy().transpose(2, 1, 0),
                    mask=torch.empty((nz, ny, nx), dtype=F64, pin_memory=True))
    if k == "poisson":
        g = grid(nx, ny, nz)
        ctx = _context(nx, ny, nz, dict(dt=1e-3, Re=RE, Sc=PR, eta=ETA, force=0.0, source=0.0,
                                        tbot=0.0, ttop=0.0, tsolid=0.0),
                       torch.zeros((nz, ny, nx), dtype=F64, device="cuda"))
        return dict(kind=k, ctx=ctx, rhs=_pinned(_wrap_samples(_poisson_input(g, case, seed))),
                    out=_buffers(shape, ("phi",)))
    if k == "mkp":
        g, us, fields, dt = _mkp_input(case, seed)
        f = {n: np.asfortranarray(x.cpu().numpy().transpose(2, 1, 0)) for n, x in us.items()}
        for n, x in fields.items():
            f[n] = np.asfortranarray(x.cpu().numpy().transpose(2, 1, 0))
        for n in ("u", "v", "w", "u_ep2", "v_ep2", "w_ep2", "divu"):
            f[n] = np.zeros((nx + 2, ny + 2, nz + 2), order="F")
        return dict(kind=k, g=g, f=f, dt=dt, n=(nx, ny, nz),
                    keep={n: f[n].copy(order="F") for n in fields})
    AC, KXZ, Y = _spn_input(case, seed)
    L = lib()
    L.nse_spn_noalloc.argtypes = [C.c_int] * 3 + [C.c_void_p] * 4
    phit = torch.zeros((nz + 2, ny + 2, nx // 2 + 1, 2), dtype=F64, device="cuda")
    return dict(kind=k, L=L, n=(nx, ny, nz), AC=AC.t().contiguous(), KXZ=KXZ, Y=Y, phit=phit)


def run(st):
    k = st["kind"]
    if k == "step":
        ctx = st["ctx"]
        _load(ctx, st["host"])
        ctx.step(st["steps"])
        return _save(ctx, st["out"])
    if k == "ensemble":
        for ctx, host in zip(st["ctx"], st["host"]):
            _load(ctx, host)
        st["ens"].step(st["steps"])
        return [_save(ctx, out) for ctx, out in zip(st["ctx"], st["out"])]
    if k == "adjoint":
        ctx, adj = st["ctx"], st["adj"]
        _load(ctx, st["host"])
        J, grad = adj.gradient()
        # the ghost cells of an adjoint field are not part of the state
        init = {n: adj.initial_adjoint(n)[1:-1, 1:-1, 1:-1] for n in ("u", "T")}
        return dict(J=J, grad=grad, **init)
    if k == "levelset":
        phi = st["ctx"].levelset(st["phi0"], nnn=st["sweeps"], dtau=1.0e-3, width=1.5)
        st["ctx"].download_ptr("cellvalue", st["mask"].data_ptr())
        return dict(phi=phi, mask=st["mask"])
    if k == "poisson":
        st["ctx"].upload_ptr("phi", st["rhs"].data_ptr())
        st["ctx"].poisson()
        return _save(st["ctx"], st["out"])
    if k == "mkp":
        f, g = st["f"], st["g"]
        for n, x in st["keep"].items():
            f[n][...] = x
        nx, ny, nz = st["n"]
        legacy.mkp(f["p"], f["us"], f["vs"], f["ws"], st["dt"], g["dx"], g["dy"], g["dz"],
                   g["dx12"], g["dy12"], g["dz12"], RE, nx, ny, nz, 1, f["u_ta"], f["v_ta"],
                   f["w_ta"], f["u_ep2"], f["v_ep2"], f["w_ep2"], f["divu"], f["u"], f["v"],
                   f["w"], XL, ZL)
        return {n: f[n] for n in ("u", "v", "w", "p", "u_ta", "v_ta", "w_ta", "u_ep2", "v_ep2",
                                  "w_ep2")}
    st["phit"].copy_(st["Y"])  # the next right-hand side, solved in place
    if st["L"].nse_spn_noalloc(*st["n"], st["AC"].data_ptr(), st["KXZ"].data_ptr(),
                               st["phit"].data_ptr(), torch.cuda.current_stream().cuda_stream):
        raise RuntimeError("nse_spn_noalloc failed")
    return st["phit"]


def _load(ctx, host):
    """a job's start: fields up, initial projection, histories, step counter 1"""
    for n, x in host.items():
        ctx.upload_ptr(n, x.data_ptr())
    ctx.project()
    ctx.step_index = 1
    ctx.start()


def _save(ctx, out):
    for n, x in out.items():
        ctx.download_ptr(n, x.data_ptr())
    return out


# ------------------------------------------------------- the job in 64 bits
def V(a, di=0, dj=0, dk=0):
    """interior of a padded tensor shifted by (di, dj, dk) cells"""
    nz, ny, nx = (n - 2 for n in a.shape)
    return a[1 + dk:nz + 1 + dk, 1 + dj:ny + 1 + dj, 1 + di:nx + 1 + di]


def _periodic(a):
    a = torch.cat([a[..., -1:], a, a[..., :1]], dim=2)
    return torch.cat([a[-1:], a, a[:1]], dim=0)


def bc_u(x):
    """u, w: no slip at the walls, periodic in x and z"""
    return _periodic(torch.cat([-x[:, :1], x, -x[:, -1:]], dim=1))


def bc_v(x):
    """v lives on the wall faces j = 0 and ny, where it is zero"""
    z = torch.zeros_like(x[:, :1])
    return _periodic(torch.cat([z, x[:, :-1], z, z], dim=1))


def bc_T(x, tb, tt):
    return _periodic(torch.cat([2.0 * tb - x[:, :1], x, 2.0 * tt - x[:, -1:]], dim=1))


def bc_p(x):
    return _periodic(torch.cat([x[:, :1], x, x[:, -1:]], dim=1))


class _Grid:
    """spacings shaped to broadcast along their axis; d(name, o): entries 1+o..n+o"""

    def __init__(self, g):
        self.t = {k: _t(v) for k, v in g.items()}
        self.shape = {"x": (1, 1, -1), "y": (1, -1, 1), "z": (-1, 1, 1)}

    def __call__(self, name, o=0):
        a = self.t[name]
        return a[1 + o:len(a) - 1 + o].view(self.shape[name[1]])


AXIS = {"x": 2, "y": 1, "z": 0}
UNIT = {"x": (1, 0, 0), "y": (0, 1, 0), "z": (0, 0, 1)}


def _neg(e):
    return tuple(-q for q in e)


def convect(G, f, comp, dt, force):
    """advection of velocity component comp in conservative form"""
    a, fa = comp, f[comp]
    tot = 0.0
    for b in "xyz":
        e, ne = UNIT[b], _neg(UNIT[b])
        c = V(fa)
        if b == a:
            t = ((c + V(fa, *e)) ** 2 - (V(fa, *ne) + c) ** 2) / G("d" + a + "12")
        else:
            ea = UNIT[a]
            gp = V(f[b], *ea) * G("d" + a, 1) + V(f[b]) * G("d" + a)
            gm = V(f[b], *[p + q for p, q in zip(ea, ne)]) * G("d" + a, 1) + V(f[b], *ne) * G("d" + a)
            t = (gp * (V(fa, *e) + c) - gm * (c + V(fa, *ne))) / G("d" + a + "12") / G("d" + b)
        tot = tot - t
    return 0.25 * tot * dt + (force * dt if a == "x" else 0.0)


def convect_T(G, f, T, dt, source):
    tot = 0.0
    for a in "xyz":
        e, ne = UNIT[a], _neg(UNIT[a])
        d = "d" + a
        lo = (V(T, *ne) * G(d) + V(T) * G(d, -1)) * V(f[a], *ne) / 2.0 / G(d + "12", -1)
        hi = (V(T) * G(d, 1) + V(T, *e) * G(d)) * V(f[a]) / 2.0 / G(d + "12")
        tot = tot - (hi - lo) / G(d)
    return tot * dt + source * dt


def laplace(G, f, stag):
    """second differences; along `stag` the points are the faces"""
    tot = 0.0
    for a in "xyz":
        e, d, d12 = UNIT[a], "d" + a, "d" + a + "12"
        up, dn = V(f, *e) - V(f), V(f) - V(f, *_neg(e))
        if a == stag:
            tot = tot + (up / G(d, 1) - dn / G(d)) / G(d12)
        else:
            tot = tot + (up / G(d12) - dn / G(d12, -1)) / G(d)
    return tot


def face_masks(c1):
    out = {}
    for a in "xyz":
        ax = AXIS[a]
        n = c1.shape[ax]
        lo, hi = c1.narrow(ax, 0, n - 1), c1.narrow(ax, 1, n - 1)
        out[a] = torch.cat([0.5 * (lo + hi), c1.narrow(ax, n - 1, 1)], dim=ax)
    return out


def _thomas(lo, di, up):
    """elimination factors of tridiagonal systems along dim 0"""
    n = di.shape[0]
    w, inv = torch.empty_like(di), torch.empty_like(di)
    inv[0] = 1.0 / di[0]
    for i in range(1, n):
        w[i] = lo[i] * inv[i - 1]
        inv[i] = 1.0 / (di[i] - w[i] * up[i - 1])
    return w, inv


def _sweep(w, inv, up, r):
    x = r.clone()
    n = x.shape[0]
    for i in range(1, n):
        x[i].addcmul_(w[i], x[i - 1], value=-1.0)
    x[n - 1].mul_(inv[n - 1])
    for i in range(n - 2, -1, -1):
        x[i].addcmul_(up[i], x[i + 1], value=-1.0).mul_(inv[i])
    return x


class _System:
    """tridiagonal (periodic: with corners) systems along dim 0, one per column"""

    def __init__(self, lo, di, up, periodic):
        lo, di, up = (t.detach() for t in (lo, di, up))
        self.periodic = periodic
        if periodic:
            gam = -di[0]
            d = di.clone()
            d[0] = d[0] - gam
            d[-1] = d[-1] - lo[0] * up[-1] / gam
            self.w, self.inv = _thomas(lo, d, up)
            e = torch.zeros_like(di)
            e[0], e[-1] = gam, up[-1]
            self.z = _sweep(self.w, self.inv, up, e)
            self.q = lo[0] / gam
            self.den = 1.0 + self.z[0] + self.q * self.z[-1]
        else:
            self.w, self.inv = _thomas(lo, di, up)
        self.up = up

    def solve(self, r):
        x = _sweep(self.w, self.inv, self.up, r)
        if self.periodic:
            x = torch.addcmul(x, (x[0] + self.q * x[-1]) / self.den, self.z, value=-1.0)
        return x


def _transposed(lo, di, up, periodic):
    lt, ut = torch.roll(up, 1, 0), torch.roll(lo, -1, 0)
    if not periodic:
        lt[0], ut[-1] = 0.0, 0.0
    return _System(lt, di, ut, periodic)


class _LineSolve(torch.autograd.Function):
    """x = A^-1 r with the derivative by r and by A's three diagonals"""

    @staticmethod
    def forward(ctx, r, lo, di, up, line):
        x = line.system.solve(r)
        ctx.line = line
        ctx.save_for_backward(x)
        return x

    @staticmethod
    def backward(ctx, xb):
        (x,) = ctx.saved_tensors
        line = ctx.line
        if line.system_t is None:
            line.system_t = _transposed(line.lo.detach(), line.di.detach(), line.up.detach(),
                                        line.system.periodic)
        y = line.system_t.solve(xb.contiguous())
        if not ctx.needs_input_grad[2]:
            return y, None, None, None, None
        xm, xp = torch.roll(x, 1, 0), torch.roll(x, -1, 0)
        if not line.system.periodic:
            xm[0], xp[-1] = 0.0, 0.0
        return y, -y * xm, -y * x, -y * xp, None


class _Line:
    """one implicit pass along an axis: 1 + dt*eta*c scales the diffusion
    operator of (f, T); walls in y (ghost sums ft, fb; v: zero), periodic else"""

    def __init__(self, G, par, axis, stag, c, ft=0.0, fb=0.0, temp=False):
        self.axis, d, d12 = AXIS[axis], "d" + axis, "d" + axis + "12"
        beta = par["dt"] / par["Re"] / 2.0 / (par["Sc"] if temp else 1.0)
        alpha = 1.0 + par["dt"] * par["eta"] * c
        v_rows = stag == "y" and not temp  # v: rows and lines 1..ny-1
        if v_rows and axis != "y":
            alpha = alpha[:, :-1]
        if axis == "y":
            if v_rows:
                lo, up = 1.0 / G(d) / G(d12), 1.0 / G(d, 1) / G(d12)
                lo, up, alpha = lo[:, :-1], up[:, :-1], alpha[:, :-1]
            else:
                lo, up = 1.0 / G(d12, -1) / G(d), 1.0 / G(d12) / G(d)
        elif temp:
            lo, up = 1.0 / G(d12, -1) / G(d), 1.0 / G(d12) / G(d)
        else:
            lo, up = 1.0 / G(d) / G(d12), 1.0 / G(d, 1) / G(d12)
        self.v_rows = v_rows
        s = beta / alpha
        lo, di, up = -s * lo, 1.0 + s * (lo + up), -s * up
        lo, di, up = (self._flat(t) for t in (lo, di, up))
        self.shift = None
        if axis == "y" and not v_rows:  # x0 = ft - x1, x(n+1) = fb - x(n)
            di = di + _ends(lo, up, -1.0, -1.0)
            if ft != 0.0 or fb != 0.0:
                self.shift = _ends(lo, up, -ft, -fb)
        self.lo, self.di, self.up = lo, di, up
        self.system, self.system_t = _System(lo, di, up, axis != "y"), None

    def _flat(self, x):
        return x.movedim(self.axis, 0).reshape(x.shape[self.axis], -1)

    def __call__(self, x):
        y = x[:, :-1] if self.v_rows else x
        m = y.movedim(self.axis, 0)
        r = m.reshape(m.shape[0], -1)
        if self.shift is not None:
            r = r + self.shift
        out = _LineSolve.apply(r, self.lo, self.di, self.up, self)
        out = out.view(m.shape).movedim(0, self.axis)
        return torch.cat([out, x[:, -1:]], dim=1) if self.v_rows else out


def _ends(lo, up, a, b):
    """a*lo in the first row, b*up in the last, zero between"""
    z = torch.zeros_like(lo[1:-1])
    return torch.cat([a * lo[:1], z, b * up[-1:]], dim=0)


class _Poisson:
    def __init__(self, g):
        self.AC, self.KXZ = _coeffs(g)
        ny = self.AC.shape[0]
        H, nz = self.KXZ.shape[1], self.KXZ.shape[0] - 1
        k = self.KXZ[:nz].reshape(1, -1)
        a, b, c = (self.AC[:, q:q + 1] for q in range(3))
        lo, up = a.expand(ny, H * nz).clone(), c.expand(ny, H * nz).clone()
        di = b - k
        di[0] += lo[0]
        di[-1] += up[-1]
        lo[0], up[-1] = 0.0, 0.0
        di[:, 0], lo[:, 0], up[:, 0] = 1.0, 0.0, 0.0
        self.lo, self.di, self.up = (t.repeat_interleave(2, dim=1) for t in (lo, di, up))
        self.system, self.system_t = _System(self.lo, self.di, self.up, False), None
        # mean mode: phi_1 = 0 and the rows 1..ny-1 marched upwards
        M = torch.zeros((ny - 1, ny), dtype=F64, device=k.device)
        i = torch.arange(ny - 1, device=k.device)
        M[i, i + 1], M[i, i] = self.AC[:-1, 2], self.AC[:-1, 1]
        M[i[1:], i[1:] - 1] = self.AC[1:-1, 0]
        self.M = M[:, 1:].contiguous()

    def spectral(self, Y):
        """(nz, ny, H) complex -> solved, the mean mode left as it is"""
        nz, ny, H = Y.shape
        r = torch.view_as_real(Y.permute(1, 0, 2).reshape(ny, nz * H).contiguous())
        x = _LineSolve.apply(r.reshape(ny, -1), self.lo, self.di, self.up, self)
        x = torch.view_as_complex(x.view(ny, nz * H, 2).contiguous())
        return x.view(ny, nz, H).permute(1, 0, 2)

    def __call__(self, rhs):
        """interior right-hand side -> interior phi"""
        nz, ny, nx = rhs.shape
        # sample 0 is cell n in x and z
        s = torch.roll(rhs, (1, 1), (0, 2))
        Y = torch.fft.rfft2(s, dim=(0, 2)) / (nx * nz)
        X = self.spectral(Y)
        m = torch.linalg.solve_triangular(self.M, Y[0, :-1, 0].real.reshape(-1, 1), upper=False)
        mean = torch.cat([torch.zeros_like(m[:1, 0]), m[:, 0]])
        keep = torch.ones(X.shape[0::2], dtype=F64, device=X.device)
        keep[0, 0] = 0.0
        X = X * keep[:, None, :]
        s = torch.fft.irfft2(X, s=(nz, nx), dim=(0, 2)) * (nx * nz) + mean[None, :, None]
        return torch.roll(s, (-1, -1), (0, 2))


def phi_padded(phi):
    """ghosts of phi as S2P and PHIBC leave them (edges of the y ghosts unset)"""
    P = bc_p(phi)
    P[:, 0, -1], P[:, -1, -1] = 0.0, 0.0
    for k in (0, -1):
        P[k, 0], P[k, -1] = 0.0, 0.0
    return P


def mkp(G, solve, us, vs, ws, dt):
    """projection of padded u*, v*, w*: interior u, v, w, dt*grad phi, phi"""
    rhs = ((V(us) - V(us, -1)) / G("dx") + (V(vs) - V(vs, 0, -1)) / G("dy") +
           (V(ws) - V(ws, 0, 0, -1)) / G("dz")) / dt
    phi = solve(rhs)
    P = bc_p(phi)
    gr = [dt * ((V(P, *UNIT[a]) - phi) / G("d" + a + "12")) for a in "xyz"]
    return [V(f) - q for f, q in zip((us, vs, ws), gr)], gr, phi


def _faces(G, old, star, P, axis, dt):
    """old with its entries 0..n replaced by star - dt * dP/d(axis)"""
    out = old.clone()
    c = (slice(0, -1),) * 3
    sh = [slice(0, -1)] * 3
    sh[AXIS[axis]] = slice(1, None)
    d12 = G.t["d" + axis + "12"][:-1].view(G.shape[axis])
    out[c] = star[c] - dt * ((P[tuple(sh)] - P[c]) / d12)
    return out


class Flow:
    """the time stepping of a penalised channel, interior state as tensors"""

    def __init__(self, g, par, c1):
        self.G, self.par, self.c1 = _Grid(g), par, c1
        self.c = face_masks(c1)
        self.solve = _Poisson(g)
        G = self.G
        L = lambda axis, stag, c, **kw: _Line(G, par, axis, stag, c, **kw)  # noqa: E731
        self.lines = {a: [L(b, a if a == "y" else "", self.c[a]) for b in "yzx"] for a in "xyz"}
        self.lines["T"] = [L("y", "", c1, ft=2.0 * par["tbot"], fb=2.0 * par["ttop"], temp=True),
                           L("x", "", c1, temp=True), L("z", "", c1, temp=True)]

    def project(self, f):
        """initial projection; starts the histories"""
        us, vs, ws = bc_u(f["u"]), bc_v(f["v"]), bc_u(f["w"])
        (u, v, w), gr, phi = mkp(self.G, self.solve, us, vs, ws, self.par["dt"])
        return dict(u=u, v=v, w=w, T=f["T"], p=phi, ta=gr, pre=[u, v, w, f["T"]])

    def step(self, s, l, keep=False):
        G, p, c1 = self.G, self.par, self.c1
        dt, eta = p["dt"], p["eta"]
        f = {"x": bc_u(s["u"]), "y": bc_v(s["v"]), "z": bc_u(s["w"])}
        T = bc_T(s["T"], p["tbot"], p["ttop"])
        a1, a2 = (1.0, 0.0) if l == 1 else (1.5, -0.5)
        star, pre = {}, []
        for i, a in enumerate("xyz"):
            cv = convect(G, f, a, dt, p["force"])
            pre.append(cv)
            r = V(f[a]) + a1 * cv + a2 * s["pre"][i] + dt / p["Re"] / 2.0 * laplace(G, f[a], a) + \
                eta * self.c[a] * s["ta"][i] * dt
            r = r / (1.0 + eta * self.c[a] * dt)
            for line in self.lines[a]:
                r = line(r)
            star[a] = r
        cv = convect_T(G, f, T, dt, p["source"])
        pre.append(cv)
        r = V(T) + a1 * cv + a2 * s["pre"][3] + dt / p["Re"] / p["Sc"] / 2.0 * laplace(G, T, "")
        r = (r + eta * c1 * dt * p["tsolid"]) / (1.0 + eta * c1 * dt)
        for line in self.lines["T"]:
            r = line(r)
        st = {"x": bc_u(star["x"]), "y": bc_v(star["y"]), "z": bc_u(star["z"])}
        (u, v, w), gr, phi = mkp(G, self.solve, st["x"], st["y"], st["z"], dt)
        out = dict(u=u, v=v, w=w, T=r, p=phi, ta=gr, pre=pre)
        if keep:  # the padded fields as the program reads them back
            P = phi_padded(phi)
            full = {n: _faces(G, f[a], st[a], P, a, dt) for n, a in zip("uvw", "xyz")}
            full["p"] = bc_p(s["p"])
            full["p"][1:-1, 1:-1, 1:-1] = phi
            full["T"] = bc_T(r, p["tbot"], p["ttop"])
            out["full"] = full
        return out


def _exact_steps(g, f, c1, par, steps):
    with torch.no_grad():
        flow = Flow(g, par, c1)
        s = flow.project(f)
        for l in range(1, steps + 1):
            s = flow.step(s, l, keep=l == steps)
    return {n: s["full"][n] for n in OUT}


def _exact_adjoint(case, seed):
    g, f, c1, par = channel(case["nx"], case["ny"], case["nz"], seed, case["obstacle"],
                            case["t_bot"])
    with torch.no_grad():
        s = Flow(g, par, c1).project(f)
    c1.requires_grad_(True)
    leaf = {n: s[n].clone().requires_grad_(True) for n in ("u", "T")}
    s = dict(s, **leaf)
    flow = Flow(g, par, c1)
    N, n0 = case["steps"], max(1, case["steps"] // 2)
    area = _t(g["dx"][1:-1])[None, :] * _t(g["dz"][1:-1])[:, None] / (XL * ZL)
    J = 0.0
    for l in range(1, N + 1):
        s = flow.step(s, l)
        if l >= n0:
            J = J + (area * (2.0 * s["T"][:, 0] - 2.0 * par["tbot"])).sum() / g["dy12"][0] / (N - n0 + 1)
    grads = torch.autograd.grad(J, [c1, leaf["u"], leaf["T"]])
    grad, u, T = (t.permute(2, 1, 0).cpu().numpy() for t in grads)
    return dict(J=float(J.detach()), grad=grad, u=u, T=T)


def _exact_levelset(case, seed):
    g, phi0 = _levelset_input(case, seed)
    G = _Grid(g)
    sgn, pos = torch.sign(phi0), phi0 > 0.0
    phi, P = phi0, _pad(phi0)  # the first sweep sees the ghosts of the input
    for _ in range(case["sweeps"] + 1):
        tot = 0.0
        for a in "xyz":
            d = "d" + a
            lo = (phi - V(P, *_neg(UNIT[a]))) / G(d + "12", -1)
            hi = (V(P, *UNIT[a]) - phi) / (G("dx") if a == "x" else G(d + "12"))
            lo, hi = torch.where(pos, lo, -lo), torch.where(pos, hi, -hi)
            tot = tot + torch.maximum(lo.clamp(min=0.0) ** 2, hi.clamp(max=0.0) ** 2)
        phi = phi - 1.0e-3 * sgn * (torch.sqrt(tot) - 1.0)
        P = torch.nn.functional.pad(phi[None, None], (1,) * 6, mode="replicate")[0, 0]
    return dict(phi=P.cpu().numpy().transpose(2, 1, 0), mask=_smooth_mask(g, phi, 1.5))


def _exact_mkp(case, seed):
    g, us, old, dt = _mkp_input(case, seed)
    G = _Grid(g)
    solve = _Poisson(g)
    _, gr, phi = mkp(G, solve, us["us"], us["vs"], us["ws"], dt)
    P = phi_padded(phi)
    out = {}
    for n, a, s in zip("uvw", "xyz", ("us", "vs", "ws")):
        out[n] = _faces(G, torch.zeros_like(P), us[s], P, a, dt)
        out[n + "_ta"] = _faces(G, old[n + "_ta"], torch.zeros_like(P), P, a, -dt)
    p = old["p"].clone()
    p[1:-1, 1:-1, 1:-1] = phi
    out["p"] = p
    for n, a in zip("uvw", "xyz"):
        out[n + "_ep2"] = _pad(-dt * (V(p, *UNIT[a]) - V(p)) / G("d" + a + "12") +
                               V(old[n + "_ta"]))
    return {n: x.cpu().numpy().transpose(2, 1, 0) for n, x in out.items()}


def exact(case, seed):
    """what `run` returns, in FP64 torch without the library"""
    k = case["kind"]
    if k == "step":
        g, f, c1, par = channel(case["nx"], case["ny"], case["nz"], seed, case["obstacle"],
                                case["t_bot"])
        return _exact_steps(g, f, c1, par, case["steps"])
    if k == "ensemble":
        out = []
        for nx, ny, nz, Re, s in _ensemble_specs(case, seed):
            out.append(_exact_steps(*channel(nx, ny, nz, s, "boxes", 1.0, Re), case["steps"]))
        return out
    if k == "adjoint":
        return _exact_adjoint(case, seed)
    if k == "levelset":
        return _exact_levelset(case, seed)
    if k == "mkp":
        with torch.no_grad():
            return _exact_mkp(case, seed)
    with torch.no_grad():
        g = grid(case["nx"], case["ny"], case["nz"])
        if k == "poisson":
            return {"phi": phi_padded(_Poisson(g)(_poisson_input(g, case, seed)))}
        _, _, Y = _spn_input(case, seed)
        nz, ny = case["nz"], case["ny"]
        out = Y.clone()
        out[:nz, 1:ny + 1] = torch.view_as_real(
            _Poisson(g).spectral(torch.view_as_complex(Y[:nz, 1:ny + 1].contiguous())).contiguous())
        return out
