"""Timed workloads of the wind solver, through its public entry points, over the
sizes and options that it is used with.

Every case is a plain dict; ``kind`` says which path it takes:

  update     one steady-state wind update: divergence, the V-cycle-preconditioned
             solve from lambda = 0 to 1e-9, the correction of u, v, w
  flexible   the same with FGMRES(30) and the composite learned preconditioner
  batch      many uneven subdomains solved by one graph launch, every fourth one
             with the learned preconditioner
  plain      a fixed number of the reference's Jacobi-preconditioned BiCGStab
             iterations on a given right-hand side (the solver-logged residuals
             that the learned preconditioner is trained on)
  calibrate  the 27-colour calibration of the projection operator and its
             coefficients
  precond    one V-cycle and the residual it leaves (z = M r, A z)
  learned    the U-Net applied to a residual
  train      one optimiser step of the U-Net: forward and backward passes over
             a batch, Adam
  stability  what precedes and follows a solve in update_winds: stability, alpha
             and its smoothing, the w predictor, the divergence, the real w

Inputs are seeded Gaussian-hill terrains with Gal-Chen metrics, log-profile
winds with noise, and an exponential density, made on the GPU (the rules of
hicar_b200.cases).  ``exact`` restates each path in 64-bit torch.
"""
import ctypes
import math
import random
from types import SimpleNamespace

import numpy as np
import torch

from hicar_b200 import _capi, batch, learned, train_unet
from hicar_b200.domain import DeviceDomain, ptr
from hicar_b200.wind_iterative import WindOptions

DX = 250.0
LR = 2e-3         # of the training step
TOL = 1e-9        # of the solves: the winds then agree to FP32 rounding
ITERATIONS = 16   # iterations a V-cycle-preconditioned solve to TOL takes, for work()
NSECT = 72        # wind-direction sectors of the blocking heights
CYCLE = learned.MG_CYCLE
# offsets (dk, dj, di) of the coefficients A..O
OFF = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 0, 1), (0, 0, -1), (0, 1, 0), (0, -1, 0), (1, 0, 1), (1, 0, -1),
       (-1, 0, 1), (-1, 0, -1), (1, 1, 0), (1, -1, 0), (-1, 1, 0), (-1, -1, 0)]
SLOT = {o: q for q, o in enumerate(OFF)}
# (cin, cout) of the U-Net's convolutions a..g
CONVS = [(16, 16), (16, 32), (32, 32), (32, 32), (32, 16), (16, 16), (16, 16)]


def listed():
    return [
        # a small nest, updated every model step: latency
        dict(name="update_64x64x20", kind="update", nx=64, ny=64, nz=20, krylov="f64", density=True, alpha="const"),
        # a nest of odd extents with varying stability
        dict(name="update_181x157x33", kind="update", nx=181, ny=157, nz=33, krylov="f64", density=True,
             alpha="smooth"),
        # a regional domain, FP32 Krylov vectors
        dict(name="update_512x512x48", kind="update", nx=512, ny=512, nz=48, krylov="mixed", density=True,
             alpha="const"),
        # the largest domain of the benchmark
        dict(name="update_1024x1024x64", kind="update", nx=1024, ny=1024, nz=64, krylov="mixed", density=True,
             alpha="smooth"),
        # flexible outer loop with the trained network
        dict(name="flexible_256x256x48", kind="flexible", nx=256, ny=256, nz=48, density=True, alpha="const"),
        # an ensemble of nests
        dict(name="batch_12", kind="batch", count=12, lo=96, hi=256, step=32, nz_lo=20, nz_hi=32, pick=0),
        # the default (reference) method
        dict(name="plain_512x512x48", kind="plain", nx=512, ny=512, nz=48, iterations=16, density=True,
             alpha="const"),
        # after every change of alpha or terrain
        dict(name="calibrate_256x256x48", kind="calibrate", nx=256, ny=256, nz=48, density=True, alpha="smooth"),
        # building training pairs, checking residuals; also the preconditioner alone
        dict(name="precond_384x320x40", kind="precond", nx=384, ny=320, nz=40, density=True, alpha="const"),
        # the learned correction on a domain larger than its training set's
        dict(name="learned_512x512x48", kind="learned", nx=512, ny=512, nz=48, density=True, alpha="const"),
        # the network's training configuration
        dict(name="train_128x128x32", kind="train", nx=128, ny=128, nz=32, samples=4),
        # the per-step work around the solve
        dict(name="stability_256x256x48", kind="stability", nx=256, ny=256, nz=48, density=True, alpha="const"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi, cells):
    while True:
        nx, ny, nz = _log_int(rng, lo, hi), _log_int(rng, lo, hi), rng.randint(12, 64)
        if nx * ny * nz <= cells:
            return dict(nx=nx, ny=ny, nz=nz)


def draw(rng):
    kind = rng.choices(["update", "flexible", "batch", "plain", "calibrate", "precond", "learned", "train",
                        "stability"], [10, 2, 2, 3, 3, 3, 3, 3, 2])[0]
    c = dict(kind=kind)
    if kind == "batch":
        lo = rng.randrange(64, 129, 16)
        return dict(c, count=rng.randint(4, 12), lo=lo, hi=lo + rng.randrange(32, 129, 32), step=rng.choice([7, 32]),
                    nz_lo=16, nz_hi=rng.randrange(20, 37, 4), pick=rng.randint(1, 10 ** 6))
    if kind == "train":
        return dict(c, **_grid(rng, 48, 192, 10 ** 6), samples=rng.randint(1, 4))
    lo, hi, cells = {"update": (48, 768, 24 * 10 ** 6), "flexible": (64, 320, 4 * 10 ** 6),
                     "plain": (48, 640, 13 * 10 ** 6), "calibrate": (48, 512, 8 * 10 ** 6),
                     "precond": (48, 640, 13 * 10 ** 6), "learned": (64, 640, 13 * 10 ** 6),
                     "stability": (48, 384, 4 * 10 ** 6)}[kind]
    c.update(_grid(rng, lo, hi, cells))
    c["density"] = rng.random() < 0.75
    c["alpha"] = rng.choice(["const", "smooth"])
    if kind == "update":
        c["krylov"] = rng.choice(["f64", "mixed"])
    if kind == "plain":
        c["iterations"] = rng.randint(4, 16)
    return c


# ---- inputs -----------------------------------------------------------------------
def _shapes(c):
    """The subdomain shapes of a batch."""
    r = random.Random(c["pick"])
    side = lambda: r.randrange(c["lo"], c["hi"] + 1, c["step"])  # noqa: E731
    return [dict(nx=side(), ny=side(), nz=r.randrange(c["nz_lo"], c["nz_hi"] + 1, 4), density=True, alpha="const")
            for _ in range(c["count"])]


def _fields(c, seed):
    """Terrain, metrics, density, alpha and winds of a case: FP32 CUDA tensors in
    the solver's layouts, (ny, nz, nx) and the face forms."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    rng = random.Random(seed * 7919 + 1)
    gen = torch.Generator("cuda").manual_seed(seed)
    f64 = dict(dtype=torch.float64, device="cuda")
    xs, ys = torch.arange(nx, **f64) * DX, torch.arange(ny, **f64) * DX
    h = torch.zeros((ny, nx), **f64)
    # at most 20 hills on 192 x 192 columns
    for _ in range(60 if nx * ny > 640 * 640 else min(20, max(4, nx * ny // 1843))):
        xc, yc = rng.uniform(0, (nx - 1) * DX), rng.uniform(0, (ny - 1) * DX)
        height, sigma = rng.uniform(200, 2000), rng.uniform(1000, 10000) / math.sqrt(2 * math.log(2))
        sigma = max(sigma, 1.5 * height)  # slopes up to 0.4 a hill, as on a grid of 250 m
        h += height * torch.outer(torch.exp(-(ys - yc) ** 2 / (2 * sigma ** 2)),
                                  torch.exp(-(xs - xc) ** 2 / (2 * sigma ** 2)))
    h = h.float()
    nominal = torch.clamp(20.0 * 1.1 ** torch.arange(nz, **f64), max=500.0)
    dz = (nominal * ((h.max().double() + nominal.sum()) / nominal.sum())).float()
    jac2 = (dz.sum() - h) / dz.sum()
    jac = jac2[:, None, :].expand(ny, nz, nx).contiguous()
    agl = (torch.cumsum(dz, 0) - dz / 2)[None, :, None] * jac  # heights of the mass levels above ground
    z = h[:, None, :] + agl

    def faces(a, dim):
        """Face means along dim, the edge cells' values on the outer faces."""
        n = a.shape[dim]
        return torch.cat([a.narrow(dim, 0, 1), (a.narrow(dim, 1, n - 1) + a.narrow(dim, 0, n - 1)) / 2,
                          a.narrow(dim, n - 1, 1)], dim).contiguous()

    def slopes(dim):
        """Centred slopes on cells (one-sided at the edges) and on faces."""
        n = z.shape[dim]
        a = [z.narrow(dim, q, 1) for q in (0, 1, 2)] + [z.narrow(dim, n - q, 1) for q in (1, 2, 3)]
        cell = torch.cat([(-3 * a[0] + 4 * a[1] - a[2]) / (2 * DX),
                          (z.narrow(dim, 2, n - 2) - z.narrow(dim, 0, n - 2)) / (2 * DX),
                          (3 * a[3] - 4 * a[4] + a[5]) / (2 * DX)], dim)
        at = lambda q: cell.narrow(dim, q, 1)  # noqa: E731
        face = torch.cat([1.5 * at(0) - 0.5 * at(1), (z.narrow(dim, 1, n - 1) - z.narrow(dim, 0, n - 1)) / DX,
                          1.5 * at(n - 1) - 0.5 * at(n - 2)], dim)
        return cell.contiguous(), face.contiguous()

    dzi = dz[None, :, None] * jac
    jw = torch.ones_like(jac)
    jw[:, :-1] = (dzi[:, 1:] * jac[:, :-1] + dzi[:, :-1] * jac[:, 1:]) / (dzi[:, :-1] + dzi[:, 1:])
    dzdx, dzdx_u = slopes(2)
    dzdy, dzdy_v = slopes(0)
    one = lambda *s: torch.ones(s, device="cuda")  # noqa: E731
    density = 1.2 * torch.exp(-z / 8000) if c["density"] else torch.ones_like(jac)
    speed, theta = rng.uniform(5, 15), rng.uniform(0, 2 * math.pi)
    profile = lambda a: speed * torch.log(torch.clamp(a, min=0.2) / 0.1) / math.log(1000.0)  # noqa: E731
    noise = lambda s: torch.randn(s, generator=gen, device="cuda")  # noqa: E731
    u = profile(faces(agl, 2)) * math.cos(theta) + noise((ny, nz, nx + 1))
    v = profile(faces(agl, 0)) * math.sin(theta) + noise((ny + 1, nz, nx))
    alpha = torch.ones_like(jac)
    if c["alpha"] == "smooth":
        x, y, k = (torch.arange(n, device="cuda") / n for n in (nx, ny, nz))
        f = torch.zeros_like(jac)
        for _ in range(8):
            kx, ky, phase = rng.randint(1, 3), rng.randint(1, 3), rng.uniform(0, 2 * math.pi)
            f += (rng.gauss(0, 1) * torch.cos(2 * math.pi * (kx * x[None, None, :] + ky * y[:, None, None]) + phase)
                  * torch.exp(-rng.uniform(0.5, 3.0) * k[None, :, None]))
        alpha = 0.3 + 0.7 * (f - f.min()) / (f.max() - f.min())
    metrics = dict(jacobian=jac, jacobian_u=faces(jac, 2), jacobian_v=faces(jac, 0), jacobian_w=jw, dzdx=dzdx,
                   dzdy=dzdy, dzdx_u=dzdx_u, dzdy_v=dzdy_v,
                   advection_dz=dz[None, :, None].expand(ny, nz, nx).contiguous(), neighbor_terrain=h,
                   mapfac_mx_u=one(ny, nx + 1), mapfac_my_v=one(ny + 1, nx), mapfac_my_u=one(ny, nx + 1),
                   mapfac_mx_v=one(ny + 1, nx), mapfac_mxy=one(ny, nx))
    return SimpleNamespace(nx=nx, ny=ny, nz=nz, dx=DX, metrics=metrics, density=density.contiguous(), z=z.contiguous(),
                           u=u.contiguous(), v=v.contiguous(), w=torch.zeros_like(jac), alpha=alpha.contiguous(),
                           gen=gen)


def _smooth_residual(nx, ny, nz, gen, passes):
    """A unit-rms residual field (ny, nz, nx) in FP64: noise, box-smoothed in x-y."""
    x = torch.randn((1, 1, ny, nz, nx), generator=gen, device="cuda", dtype=torch.float64)
    pad = torch.nn.functional.pad
    for _ in range(passes):
        x = torch.nn.functional.avg_pool3d(pad(x, (1, 1, 0, 0, 1, 1), mode="replicate"), (3, 1, 3), stride=1)
    return (x / x.square().mean().sqrt())[0, 0]


def _with_ghosts(x):
    return torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1)).contiguous()


def _residual(c, seed):
    gen = torch.Generator("cuda").manual_seed(seed + 17)
    return _with_ghosts(_smooth_residual(c["nx"], c["ny"], c["nz"], gen, 1 + seed % 4))


class Solver:
    """A calibrated solver handle and its domain, as a program keeps them per nest."""

    def __init__(self, f, c, options=None, calibrate=True):
        self.lib = _capi.load()
        self.stream = torch.cuda.current_stream().cuda_stream
        self.adv = int(c["density"])
        self.dom = DeviceDomain(nx=f.nx, ny=f.ny, nz=f.nz, dx=f.dx, nest_indx=1, metrics=f.metrics, density=f.density,
                                u_dqdt=f.u.clone(), v_dqdt=f.v.clone(), w_dqdt=f.w.clone(), wind_alpha=f.alpha)
        self.winds = (f.u, f.v, f.w)
        self.div = torch.empty((f.ny, f.nz, f.nx), device="cuda")
        self.h = ctypes.c_void_p()
        self.net = None
        g = _capi.Grid(f.nx, f.ny, f.nz, f.dx, 1)
        m = _capi.Metrics(*[ptr(f.metrics[n]) for n in _capi.METRIC_FIELDS])
        o = (options or WindOptions(windtype=0)).to_c()
        _capi.check(self.lib.hicarw_init_iter_winds(ctypes.byref(g), ctypes.byref(o), ctypes.byref(m),
                                                    _capi.MEM_DEVICE, self.stream, ctypes.byref(self.h)))
        if calibrate:
            self.calibrate()

    def call(self, name, *args):
        return _capi.check(getattr(self.lib, name)(self.h, *args), self.h)

    def rho(self):
        return ptr(self.dom.density) if self.adv else None

    def calibrate(self):
        d, leak = self.dom, ctypes.c_float()
        self.call("hicarw_calibrate_projection_operator", ptr(d.wind_alpha), self.rho(), self.adv, ptr(d.u_dqdt),
                  ptr(d.v_dqdt), ptr(d.w_dqdt), ctypes.byref(leak), _capi.MEM_DEVICE, self.stream)

    def divergence(self):
        d = self.dom
        self.call("hicarw_calc_divergence", ptr(d.u_dqdt), ptr(d.v_dqdt), ptr(d.w_dqdt), self.rho(), ptr(self.div),
                  self.adv, 0, 1, _capi.MEM_DEVICE, self.stream)

    def update(self):
        d, st = self.dom, _capi.Stats()
        d.set_winds(*self.winds)
        self.divergence()
        self.call("hicarw_reset_solution", self.stream)
        rc = self.call("hicarw_calc_iter_winds", ptr(d.wind_alpha), ptr(self.div), self.rho(), self.adv,
                       ptr(d.u_dqdt), ptr(d.v_dqdt), ptr(d.w_dqdt), _capi.MEM_DEVICE, self.stream, ctypes.byref(st))
        if rc != _capi.HICARW_OK:
            raise RuntimeError("the solve ended with status %d after %d iterations" % (rc, st.iterations))
        return dict(u=d.u_dqdt, v=d.v_dqdt, w=d.w_dqdt)

    def close(self):
        if self.h:
            self.lib.hicarw_finalize_iter_winds(self.h)
            self.h = None
        if self.net is not None:
            self.net.close()

    def __del__(self):
        self.close()


def _options(c):
    """The solve options of a case (windtype 0: no solver output on stderr)."""
    base = dict(windtype=0, advect_density=bool(c.get("density", True)), tol_rel=TOL, wind_solver_iterations=3000,
                precond=_capi.PRECOND_MG, stall_iters=50, **CYCLE)
    if c["kind"] == "flexible":
        base.update(solver=_capi.SOLVER_FGMRES, precond=_capi.PRECOND_MG_LEARNED, stall_iters=200)
    elif c["kind"] == "plain":
        base = dict(windtype=0, tol_rel=1e-30, tol_abs=0.0, wind_solver_iterations=c["iterations"])
    elif c.get("krylov") == "mixed":
        base["solver"] = _capi.SOLVER_MIXED
    return WindOptions(**base)


def _samples(c, seed):
    """Network inputs (samples, FP64 (16, ny, nz, nx)) and targets of a training
    batch: residuals of different smoothness with their operator's stencil ratios."""
    f = _fields(dict(c, density=True, alpha="const"), seed)
    coefs = _coefficients(f, True)
    ratios = coefs[1:] / coefs[0]
    out = []
    for q in range(c["samples"]):
        r = _smooth_residual(f.nx, f.ny, f.nz, f.gen, 2 * q)
        t = 0.7 * r + 0.7 * _smooth_residual(f.nx, f.ny, f.nz, f.gen, 3)
        out.append((torch.cat([r[None], ratios, torch.zeros_like(r)[None]]), t.float()))
    return out


def _stability_inputs(f):
    """Potential temperature (4 K/km with noise) and the blocking height per sector."""
    theta = 288.0 + 0.004 * f.z + 0.2 * torch.randn(f.z.shape, generator=f.gen, device="cuda")
    blocking = 3000 * torch.rand((NSECT,) + f.z.shape, generator=f.gen, device="cuda")
    w_given = 0.1 * torch.randn(f.z.shape, generator=f.gen, device="cuda")
    return theta, torch.maximum(blocking, f.metrics["advection_dz"] * f.metrics["jacobian"]), w_given


def _prepare_batch(c, seed):
    subs = []
    for q, shape in enumerate(_shapes(c)):
        f = _fields(shape, seed * 101 + q)
        host = {k: a.cpu().numpy() for k, a in f.metrics.items()}
        dom = SimpleNamespace(nx=f.nx, ny=f.ny, nz=f.nz, dx=f.dx, density=f.density.cpu().numpy(), **host)
        subs.append(SimpleNamespace(domain=dom, adv_den=True,
                                    **{k: getattr(f, k).cpu().numpy() for k in ("u", "v", "w", "alpha")}))
    return batch.BatchSolver(subs, options=_options(c), learned_every=4, learned_params=_parameters())


def _prepare_train(c, seed):
    net = learned.UNet(c["nx"], c["ny"], c["nz"])
    pairs = [(learned.to_act(x), t, 1.0 / float(t.double().square().mean())) for x, t in _samples(c, seed)]
    return SimpleNamespace(net=net, params=_parameters().cuda(), pairs=pairs)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        return c, _prepare_batch(c, seed)
    if kind == "train":
        return c, _prepare_train(c, seed)
    f = _fields(c, seed)
    s = Solver(f, c, _options(c), calibrate=kind != "calibrate")
    if kind in ("flexible", "learned"):
        s.net = learned.UNet(f.nx, f.ny, f.nz)
        s.net.set_params(_parameters())
        s.net.attach(s.h)
    if kind in ("plain", "precond", "learned"):
        s.r = _residual(c, seed)
    if kind == "calibrate":
        s.coefs = torch.empty((15, f.ny, f.nz, f.nx), device="cuda")
    if kind == "stability":
        s.z, (s.theta, s.blocking, s.w_given) = f.z, _stability_inputs(f)
        s.froude, s.ri, s.w_real = (torch.empty_like(s.div) for _ in range(3))
    return c, s


# ---- one pass ---------------------------------------------------------------------
def _run_plain(s):
    st, x = _capi.Stats(), torch.empty_like(s.r)
    s.call("hicarw_reset_solution", s.stream)
    s.call("hicarw_solve_rhs", ptr(s.r), _capi.MEM_DEVICE, s.stream, ctypes.byref(st))
    s.call("hicarw_get_lambda", ptr(x), _capi.MEM_DEVICE, s.stream)
    return x


def _run_calibrate(s):
    s.calibrate()
    s.call("hicarw_get_coefs", ptr(s.coefs), _capi.MEM_DEVICE, s.stream)
    return s.coefs


def _run_precond(s):
    z, az = torch.empty_like(s.r), torch.empty_like(s.r)
    s.call("hicarw_apply_precond", ptr(s.r), ptr(z), 0, _capi.MEM_DEVICE, s.stream)
    s.call("hicarw_apply_operator", ptr(z), ptr(az), _capi.MEM_DEVICE, s.stream)
    return dict(z=z, az=az)


def _run_stability(s):
    d, dev = s.dom, _capi.MEM_DEVICE
    u, v, w, alpha = ptr(d.u_dqdt), ptr(d.v_dqdt), ptr(d.w_dqdt), ptr(d.wind_alpha)
    s.call("hicarw_update_stability", u, v, ptr(s.z), ptr(s.theta), ptr(s.blocking), NSECT, 1, ptr(s.froude),
           ptr(s.ri), dev, s.stream)
    s.call("hicarw_calc_alpha", ptr(s.froude), alpha, 1, dev, s.stream)
    s.call("hicarw_smooth_alpha", alpha, 1, 3, dev, s.stream)
    s.call("hicarw_calc_idealized_wgrid", u, v, ptr(s.w_given), w, dev, s.stream)
    s.divergence()
    s.call("hicarw_calc_w_real", u, v, w, ptr(s.w_real), dev, s.stream)
    return dict(froude=s.froude, ri=s.ri, alpha=d.wind_alpha, w=d.w_dqdt, div=s.div, w_real=s.w_real)


def _run_train(s):
    s.net.set_params(s.params)
    s.net.zero_grads()
    for x0, target, weight in s.pairs:
        s.net.forward(x0)
        s.net.backward(target, weight)
    grads = s.net.grads()
    s.net.adam_step(LR)
    return dict(grads=grads, params=s.net.params())


def _run_batch(b):
    b.step()
    return [[d.u_dqdt, d.v_dqdt, d.w_dqdt] for d in b.domains]


RUN = dict(update=Solver.update, flexible=Solver.update, batch=_run_batch, plain=_run_plain, calibrate=_run_calibrate,
           precond=_run_precond, learned=lambda s: s.net.apply(s.h, s.r), train=_run_train, stability=_run_stability)


def run(state):
    case, s = state
    return RUN[case["kind"]](s)


def work(case):
    """Bytes and operations per cell that a pass cannot do without, in the stored
    precisions: FP32 fields and coefficients, the Krylov vectors, BF16 activations."""
    c, kind = case, case["kind"]
    if kind == "batch":
        each = [work(dict(s, kind="update", krylov="f64")) for s in _shapes(c)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    n = c["nx"] * c["ny"] * c["nz"]
    # multiplications and additions of the network: a, f, g on the full grid, b, e on a quarter, c, d on a sixteenth
    net_flops = 54 * (3 * 256 + 2 * 512 / 4 + 2 * 1024 / 16)
    net_bytes = 2 * (3 * 32 + 2 * 48 / 4 + 2 * 64 / 16)
    e = 4 if c.get("krylov") == "mixed" else 8
    cycle = 60 * 4 / 3 + 2 * e              # every level's coefficients once, the residual in, the correction out
    operator = 60 + 2 * e
    if kind in ("update", "flexible"):
        step = 2 * (cycle + operator) + 10 * e
        flops = 2 * (3 * 30 + 30) + 30
        if kind == "flexible":               # two operator applies, one cycle, one network and the Arnoldi vectors
            step = cycle + 3 * operator + net_bytes + 2 * 8 * ITERATIONS
            flops = 6 * 30 + net_flops + 4 * ITERATIONS
        return dict(bytes=n * (100 + ITERATIONS * step), flops=n * (100 + ITERATIONS * flops))
    per = dict(plain=lambda: (24 + c["iterations"] * (4 * operator + 15 * 8), c["iterations"] * 160),
               calibrate=lambda: (13 * 4 + 60, 27 * 60), precond=lambda: (cycle + operator, 5 * 30),
               learned=lambda: (60 + 16 + net_bytes, net_flops),
               train=lambda: (c["samples"] * 3 * net_bytes, c["samples"] * 3 * net_flops),
               stability=lambda: (25 * 4, 200))[kind]()
    return dict(bytes=n * per[0], flops=n * per[1])


# ---- the same in 64 bits ------------------------------------------------------------
class Exact:
    """The divergence D, the wind correction G and the operator A = 2 D G of a
    case in FP64, on (ny, nz, nx) arrays."""

    def __init__(self, f, density):
        self.f, self.density = f, density
        m = self.m = {k: a.double() for k, a in f.metrics.items()}
        self.rho = f.density.double() if density else torch.ones_like(m["jacobian"])
        dz = m["advection_dz"][0, :, 0]
        self.dzi = torch.cat([dz[:1], (dz[1:] + dz[:-1]) / 2, dz[-1:]])
        r, adz = self.rho, m["advection_dz"]
        self.rho_w = r.clone()
        self.rho_w[:, :-1] = (r[:, :-1] * adz[:, 1:] + r[:, 1:] * adz[:, :-1]) / (adz[:, :-1] + adz[:, 1:])
        self.rho_u, self.rho_v = self._faces(r, 2, 1.0, 0.0), self._faces(r, 0, 1.0, 0.0)
        self.flux_u, self.flux_v, self.flux_w = 1.0, 1.0, m["jacobian_w"]
        if density:
            self.flux_u = m["jacobian_u"] * self._faces(r, 2, 1.5, -0.5)
            self.flux_v = m["jacobian_v"] * self._faces(r, 0, 1.5, -0.5)
            self.flux_w = m["jacobian_w"] * self.rho_w

    @staticmethod
    def _faces(a, dim, p, q):
        n = a.shape[dim]
        at = lambda i: a.narrow(dim, i, 1)  # noqa: E731
        return torch.cat([p * at(0) + q * at(1), (a.narrow(dim, 1, n - 1) + a.narrow(dim, 0, n - 1)) / 2,
                          p * at(n - 1) + q * at(n - 2)], dim)

    def divergence(self, u, v, w):
        fu, fv, fw = u * self.flux_u, v * self.flux_v, w * self.flux_w
        out = (fu[:, :, 1:] - fu[:, :, :-1] + fv[1:] - fv[:-1]) / DX
        adz = self.m["advection_dz"]
        out += fw / adz
        out[:, 1:] -= fw[:, :-1] / adz[:, 1:]
        return out / self.m["jacobian"]

    def correction(self, x, alpha):
        """G x: what lambda = x (zero outside) adds to u, v and w."""
        pad = torch.nn.functional.pad
        out = []
        for dim, slope, jac, rho in ((2, "dzdx_u", "jacobian_u", self.rho_u), (0, "dzdy_v", "jacobian_v", self.rho_v)):
            e = pad(x, (1, 1, 0, 0, 0, 0) if dim == 2 else (0, 0, 0, 0, 1, 1))
            n = e.shape[dim] - 1
            lo, hi = e.narrow(dim, 0, n), e.narrow(dim, 1, n)
            mean = (lo + hi) / 2
            dl = torch.empty_like(mean)
            dl[:, 1:-1] = (mean[:, 2:] - mean[:, :-2]) / (self.dzi[2:-1] + self.dzi[1:-2])[None, :, None]
            dl[:, 0] = (mean[:, 1] - mean[:, 0]) / self.dzi[1]
            dl[:, -1] = (mean[:, -1] - mean[:, -2]) / self.dzi[-2]
            out.append(0.5 * ((hi - lo) / DX - self.m[slope] * dl / self.m[jac]) / rho)
        w = torch.zeros_like(x)
        w[:, :-1] = (0.5 * alpha[:, :-1] ** 2 * (x[:, 1:] - x[:, :-1]) / self.dzi[1:-1][None, :, None]
                     / self.m["jacobian_w"][:, :-1] / self.rho_w[:, :-1])
        return (*out, w)

    def coefficients(self, alpha):
        """The 15 coefficients of A, from the responses to 27 patterns of unit points."""
        f = self.f
        coefs = torch.zeros((15, f.ny, f.nz, f.nx), dtype=torch.float64, device="cuda")
        for cj in range(3):
            for ck in range(3):
                for ci in range(3):
                    x = torch.zeros((f.ny, f.nz, f.nx), dtype=torch.float64, device="cuda")
                    x[cj::3, ck::3, ci::3] = 1
                    t = 2 * self.divergence(*self.correction(x, alpha))
                    for q, (dk, dj, di) in enumerate(OFF):
                        at = (slice((cj - dj) % 3, None, 3), slice((ck - dk) % 3, None, 3), slice((ci - di) % 3, None, 3))
                        coefs[q][at] = t[at]
        return coefs


def _coefficients(f, density):
    return Exact(f, density).coefficients(f.alpha.double())


def _apply(coefs, x):
    """A x on the interior, x zero outside."""
    ny, nz, nx = x.shape
    e = torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))
    y = torch.zeros_like(x)
    for q, (dk, dj, di) in enumerate(OFF):
        y.addcmul_(coefs[q], e[1 + dj:1 + dj + ny, 1 + dk:1 + dk + nz, 1 + di:1 + di + nx])
    return y


class Cycle:
    """The V-cycle: V(0,1) on the finest level, W on the levels of CYCLE, column
    solves as the smoother, 2x2 x-y aggregation down to one column."""

    def __init__(self, coefs):
        self.lev = [coefs]
        while self.lev[-1].shape[1] > 1 or self.lev[-1].shape[3] > 1:
            self.lev.append(self._coarsen(self.lev[-1]))
        self.fac = [self._factors(a) for a in self.lev]

    @staticmethod
    def _sum(x):
        """Sums over the 2x2 aggregates of the first and last dimension of (..., ny, nz, nx)."""
        ny, nx = x.shape[-3], x.shape[-1]
        x = torch.nn.functional.pad(x, (0, nx % 2, 0, 0, 0, ny % 2))
        return (x[..., 0::2, :, 0::2] + x[..., 1::2, :, 0::2]) + (x[..., 0::2, :, 1::2] + x[..., 1::2, :, 1::2])

    @classmethod
    def _coarsen(cls, coefs):
        _, ny, nz, nx = coefs.shape
        out = torch.zeros((15, (ny + 1) // 2, nz, (nx + 1) // 2), dtype=torch.float64, device="cuda")
        j, k, i = (torch.arange(n, device="cuda").reshape(s) for n, s in ((ny, (-1, 1, 1)), (nz, (1, -1, 1)), (nx, (-1,))))
        for q, (dk, dj, di) in enumerate(OFF):
            inside = ((j + dj >= 0) & (j + dj < ny) & (k + dk >= 0) & (k + dk < nz) & (i + di >= 0) & (i + di < nx))
            a = torch.where(inside, coefs[q], 0.0)
            for pj in (0, 1):
                for pi in (0, 1):
                    part = a[pj::2, :, pi::2]
                    slot = SLOT[(dk, (pj + dj) // 2, (pi + di) // 2)]
                    out[slot, :part.shape[0], :, :part.shape[2]] += part
        return out

    @staticmethod
    def _factors(coefs):
        diag, up, low = coefs[0], coefs[1], coefs[2]
        nz = diag.shape[1]
        cp, mi = torch.zeros_like(diag), torch.zeros_like(diag)
        for k in range(nz):
            den = diag[:, k] - low[:, k] * cp[:, k - 1] if k else diag[:, k]
            mi[:, k] = 1 / den
            if k < nz - 1:
                cp[:, k] = up[:, k] * mi[:, k]
        return cp, mi

    def _columns(self, lev, r):
        low, (cp, mi) = self.lev[lev][2], self.fac[lev]
        y = r.transpose(0, 1).contiguous()
        low, cp, mi = low.transpose(0, 1), cp.transpose(0, 1), mi.transpose(0, 1)
        y[0] *= mi[0]
        for k in range(1, y.shape[0]):
            y[k].addcmul_(low[k], y[k - 1], value=-1).mul_(mi[k])
        for k in range(y.shape[0] - 2, -1, -1):
            y[k].addcmul_(cp[k], y[k + 1], value=-1)
        return y.transpose(0, 1)

    def _level(self, lev, r, x):
        a = self.lev[lev]
        ny, _, nx = r.shape
        for _ in range(2 if lev in CYCLE["mg_w_levels"] else 1):
            rc = self._sum(r - _apply(a, x) if x is not None else r)
            xc = self._columns(lev + 1, rc)
            if lev + 2 < len(self.lev):
                xc = self._level(lev + 1, rc, CYCLE["mg_omega"] * xc)
            up = 1.35 * xc.repeat_interleave(2, 0).repeat_interleave(2, 2)[:ny, :, :nx]
            x = up if x is None else x + up
            x = x + CYCLE["mg_omega"] * self._columns(lev, r - _apply(a, x))
        return x

    def __call__(self, r):
        return self._level(0, r, None)


def _bicgstab(a, m, b, tol, iterations):
    """Right-preconditioned BiCGStab from zero; None where it does not reach tol > 0."""
    dot = lambda p, q: (p * q).sum()  # noqa: E731
    x, r, hat, p = torch.zeros_like(b), b.clone(), b, b.clone()
    rho, target = dot(hat, r), tol * b.norm()
    for _ in range(iterations):
        ph = m(p)
        v = _apply(a, ph)
        alpha = rho / dot(hat, v)
        s = r - alpha * v
        sh = m(s)
        t = _apply(a, sh)
        omega = dot(t, s) / dot(t, t)
        x += alpha * ph + omega * sh
        r = s - omega * t
        if r.norm() <= target:
            return x
        new = dot(hat, r)
        p = r + (new / rho) * (alpha / omega) * (p - omega * v)
        rho = new
    return x if tol == 0 else None


def _solved_winds(f, density):
    """u, v, w after the correction by the solution of A x = -2 D(u, v, w)."""
    e, alpha = Exact(f, density), f.alpha.double()
    winds = [a.double() for a in (f.u, f.v, f.w)]
    a = e.coefficients(alpha)
    x = _bicgstab(a, Cycle(a), -2 * e.divergence(*winds), 1e-12, 60)
    return [None] * 3 if x is None else [w + g for w, g in zip(winds, e.correction(x, alpha))]


def _jacobi(a):
    """Two Jacobi-Richardson sweeps."""
    def apply(r):
        z = r / a[0]
        return z + (r - _apply(a, z)) / a[0]
    return apply


def _parameters():
    return torch.from_numpy(np.load(train_unet.COMPOSITE_WEIGHTS).astype(np.float32))


def _network(params, x):
    """The network's output channel 0 for features x (16, ny, nz, nx)."""
    pad = torch.nn.functional.pad
    layers, o = [], 0
    for cin, cout in CONVS:
        n = 27 * cin * cout
        layers.append((params[o:o + n].reshape(27, cin, cout), params[o + n:o + n + cout]))
        o += n + cout

    def conv(q, x):
        w, b = layers[q]
        _, ny, nz, nx = x.shape
        e = pad(x, (1, 1, 1, 1, 1, 1))
        y = b[:, None]
        for t in range(27):
            j, k, i = t // 9, t // 3 % 3, t % 3
            y = y + w[t].T @ e[:, j:j + ny, k:k + nz, i:i + nx].reshape(x.shape[0], -1)
        return y.reshape(-1, ny, nz, nx)

    def up(x, like):
        return x.repeat_interleave(2, 1).repeat_interleave(2, 3)[:, :like.shape[1], :, :like.shape[3]]

    e0 = torch.relu(conv(0, x))
    e1 = torch.relu(conv(1, Cycle._sum(e0) / 4))
    e2 = torch.relu(conv(2, Cycle._sum(e1) / 4))
    f2 = torch.relu(conv(3, e2))
    d1 = torch.relu(conv(4, up(f2, e1) + e1))
    d0 = torch.relu(conv(5, up(d1, e0)) + e0)
    return (conv(6, d0) + x)[0]


def _exact_train(c, seed):
    p = _parameters().cuda().double().requires_grad_(True)
    for x, t in _samples(c, seed):
        t = t.double()
        ((_network(p, x.to(torch.bfloat16).double()) - t).square().mean() / t.square().mean()).backward()
    g = p.grad / c["samples"]
    return dict(grads=p.grad, params=p.detach() - LR * g / (g.abs() + 1e-8))


def _exact_stability(f, c):
    e = Exact(f, c["density"])
    u, v, m = f.u.double(), f.v.double(), e.m
    _, _, given = _stability_inputs(f)

    def real(w):
        su, sv = u * m["dzdx_u"], v * m["dzdy_v"]
        out = (su[:, :, :-1] + su[:, :, 1:] + sv[:-1] + sv[1:]) / 2
        if w is not None:
            w = w * m["jacobian_w"] / 2
            out = out + w
            out[:, 1:] += w[:, :-1]
        return out

    d, adz = given.double() - real(None), m["advection_dz"]
    w = torch.zeros_like(d)
    w[:, :-1] = ((d[:, :-1] * adz[:, 1:] + d[:, 1:] * adz[:, :-1]) / (adz[:, :-1] + adz[:, 1:])
                 / m["jacobian_w"][:, :-1])
    # the sector of a wind direction and a stability at its zero are steps: no 64-bit value of what follows them
    return dict(froude=None, ri=None, alpha=None, w=w, div=e.divergence(u, v, w), w_real=real(w))


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "train":
        return _exact_train(c, seed)
    if kind == "batch":
        winds = [_solved_winds(_fields(s, seed * 101 + q), True) for q, s in enumerate(_shapes(c))]
        return winds if any(w[0] is not None for w in winds) else None
    f = _fields(c, seed)
    if kind == "stability":
        return _exact_stability(f, c)
    if kind in ("update", "flexible"):
        winds = _solved_winds(f, c["density"])
        return dict(zip("uvw", winds)) if winds[0] is not None else None
    a = _coefficients(f, c["density"])
    if kind == "calibrate":
        return a
    r = _residual(c, seed)[1:-1, 1:-1, 1:-1].contiguous()
    if kind == "plain":
        return _with_ghosts(_bicgstab(a, _jacobi(a), r, 0.0, c["iterations"]))
    if kind == "precond":
        z = Cycle(a)(r)
        return dict(z=_with_ghosts(z), az=_with_ghosts(_apply(a, z)))
    rms = r.square().mean().sqrt()
    with torch.no_grad():
        x = torch.cat([(r / rms)[None], a[1:] / a[0], torch.zeros_like(r)[None]])
        return _with_ghosts(_network(_parameters().cuda().double(), x) * rms / a[0])
