"""Performance cases: the calls a user of this framework makes, over the range of sizes and options it is used with.

A "steps" case is a run of a solver as a host program drives it through the C ABI: the velocity goes in from
page-locked f32 arrays (the element type of uploadVelocity), a few steps are advanced, and the velocity comes back.
"batch" advances many uneven domains together, "frame" is an interactive session (step, dye, rendered image), and
"predict" / "grad" are the learned pressure guess at run time and in training.  exact() restates each in 64 bits with
plain torch operations.
"""
import importlib
import math
from pathlib import Path

import numpy as np
import torch

fs = importlib.import_module("fluid-sim_gb300")
TWO_PI = 2 * math.pi
WEIGHTS = Path(fs.__file__).resolve().parent / "weights" / "guess_2048_f2.fsguess"
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def steps_case(name=None, **kw):
    c = dict(kind="steps", nx=256, ny=256, pressure="jacobi", iterations=40, advection="maccormack", precision="f32",
             tol=0.0, relative=False, relax=1.0, coarse=40, first=-1, nu=0.0, flow="modes", modes=0, band=False,
             channel=False, disks=0, steps=8)
    c.update(kw)
    if name:
        c["name"] = name
    return c


MIXED = dict(pressure="multigrid", iterations=1, precision="mixed", relax=1.2)


def listed():
    return [
        # the constructor's defaults (256^2, Jacobi 40, MacCormack, f32): the first thing a user runs, latency-bound
        steps_case("default-256"),
        # red-black smoothing on an odd, non-square grid with semi-Lagrangian advection: nothing is aligned
        steps_case("redblack-333x500", nx=333, ny=500, pressure="red-black", advection="semi-lagrangian", nu=1e-4,
                   steps=6),
        # the default solver at a display resolution
        steps_case("jacobi-1280x720", nx=1280, ny=720, nu=1e-4, disks=1, steps=4),
        # four f32 V-cycles per step with the fixed-mode forcing: the reference harness's multigrid configuration
        steps_case("mg-512", nx=512, ny=512, pressure="multigrid", iterations=4, nu=1e-4, modes=16, steps=8),
        # a small domain solved to max|div u| <= 1e-6: coarse levels and launches
        steps_case("mixed-192", nx=192, ny=192, nu=1e-4, flow="blobs", tol=1e-6, steps=8, **MIXED),
        # forced turbulence: Gaussian band forcing renewed every step, relative residual 1e-6
        steps_case("forced-1024", nx=1024, ny=1024, nu=1e-4, flow="turbulence", tol=1e-6, relative=True, band=True,
                   steps=6, **MIXED),
        # the headline workload: channel flow past disks at 2048^2, max|div u| <= 1e-6
        steps_case("channel-2048", nx=2048, ny=2048, nu=1e-4, tol=1e-6, coarse=8, first=0, channel=True, disks=5,
                   steps=6, **MIXED),
        # decaying turbulence at 4096^2 solved to max|div u| <= 1e-10: the largest working set
        steps_case("decaying-4096", nx=4096, ny=4096, nu=5e-5, flow="turbulence", tol=1e-10, steps=3, **MIXED),
        # uneven independent domains advanced by one graph launch per step
        dict(name="batch-96", kind="batch", count=96, steps=8),
        # the pressure guess as a 2048^2 solver evaluates it each step (half resolution, one image)
        dict(name="predict-1024", kind="predict", h=1024, w=1024, batch=1),
        # its training step's loss and gradients at the training configuration
        dict(name="grad-1024x4", kind="grad", h=1024, w=1024, batch=4),
        # an interactive session: step, dye, rendered image
        dict(name="frame-576", kind="frame", nx=576, iterations=4, frames=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mg_side(rng, lo, hi):
    """a multigrid side: 8..15 times a power of two (what the level hierarchy divides)"""
    while True:
        n = rng.randint(8, 15) << rng.randint(0, 8)
        if lo <= n <= hi and (n >= 512 or rng.random() < 0.6):
            return n


def draw(rng):
    kind = rng.choice(["flat", "flat", "mg", "mixed", "mixed", "batch", "predict", "grad", "frame"])
    if kind == "flat":
        return steps_case(nx=_log_int(rng, 60, 1400), ny=_log_int(rng, 60, 1400),
                          pressure=rng.choice(["jacobi", "red-black"]), iterations=rng.randint(20, 80),
                          advection=rng.choice(["maccormack", "semi-lagrangian"]), nu=rng.choice([0.0, 1e-4]),
                          disks=rng.randint(0, 2), steps=rng.randint(3, 6))
    if kind == "mg":
        n = _mg_side(rng, 64, 2048)
        return steps_case(nx=n, ny=n, pressure="multigrid", iterations=rng.randint(2, 6), nu=rng.choice([0.0, 1e-4]),
                          modes=rng.choice([0, 8, 24]), steps=rng.randint(3, 6))
    if kind == "mixed":
        n = _mg_side(rng, 64, 2880)
        return steps_case(nx=n, ny=n, nu=rng.choice([1e-4, 5e-5]), flow=rng.choice(["modes", "blobs", "turbulence"]),
                          tol=1e-6, relative=rng.random() < 0.3, coarse=rng.choice([8, 40]),
                          first=rng.choice([-1, 0]), disks=rng.randint(0, 4), steps=rng.randint(3, 6), **MIXED)
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(8, 96), steps=rng.randint(3, 8))
    if kind == "frame":
        return dict(kind="frame", nx=_mg_side(rng, 128, 1024), iterations=rng.randint(2, 5), frames=rng.randint(2, 4))
    hi = 1024 if kind == "predict" else 768
    return dict(kind=kind, h=8 * _log_int(rng, 8, hi // 8), w=8 * _log_int(rng, 8, hi // 8), batch=rng.randint(1, 4))


# ------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _curl(psi, h):
    """MAC velocity of a corner streamfunction: divergence-free on the grid"""
    return (torch.roll(psi, -1, 0) - psi) / h, -(torch.roll(psi, -1, 1) - psi) / h


def _corners(nx, ny, h):
    x = torch.arange(nx, device=DEV, dtype=torch.float64) * h
    y = torch.arange(ny, device=DEV, dtype=torch.float64) * h
    return x[None, :], y[:, None]


def _flow(c, seed, flow=None):
    """initial velocity ([ny, nx] f32 pair), and dt at CFL 0.5"""
    nx, ny = c["nx"], c["ny"]
    h = TWO_PI / nx
    rng = np.random.default_rng(seed)
    flow = flow or c["flow"]
    X, Y = _corners(nx, ny, h)
    psi = torch.zeros(ny, nx, device=DEV, dtype=torch.float64)
    if flow == "modes":  # a stream with a band of random modes
        ly = h * ny
        for _ in range(24):
            kx, ky = (int(k) for k in rng.integers(-8, 9, size=2))
            kx = kx or 3
            psi += rng.normal() * torch.sin(kx * X + ky * (TWO_PI / ly) * Y + rng.uniform(0, TWO_PI)) / (kx * kx + ky * ky)
        u, v = _curl(psi, h)
        scale = 0.1 / float(torch.maximum(u.abs().max(), v.abs().max())) if c.get("channel") else 1.0 / float(u.abs().max())
        u, v = u * scale + (1.0 if c.get("channel") else 0.3), v * scale
        if c.get("channel"):
            yu = (torch.arange(ny, device=DEV, dtype=torch.float64) + 0.5) * h
            u = u * ((yu + math.pi) % TWO_PI - math.pi).abs().gt(TWO_PI / 32)[:, None]
    else:
        k = torch.fft.fftfreq(nx, d=1.0 / nx, device=DEV, dtype=torch.float64)
        k2 = k[None, :] ** 2 + k[:, None] ** 2
        if flow == "blobs":  # 4-16 Gaussian vortices
            w = torch.zeros(ny, nx, device=DEV, dtype=torch.float64)
            for _ in range(int(rng.integers(4, 17))):
                r = float(rng.uniform(0.05, 0.15)) * TWO_PI
                cx, cy = (float(t) for t in rng.uniform(0, TWO_PI, size=2))
                dx = torch.remainder(X - cx + math.pi, TWO_PI) - math.pi
                dy = torch.remainder(Y - cy + math.pi, TWO_PI) - math.pi
                w += float(rng.normal()) / (TWO_PI * r * r) * torch.exp(-(dx * dx + dy * dy) / (2 * r * r))
            hat = torch.fft.fft2(w) / k2.clamp(min=1.0)
        else:  # random phases with E(k) ~ k^4 exp(-(k/16)^2)
            kk = k2.sqrt()
            phase = torch.rand(ny, nx, device=DEV, dtype=torch.float64, generator=_generator(seed)) * TWO_PI
            hat = torch.polar((kk * torch.exp(-(kk / 16) ** 2)).sqrt(), phase)
        hat[0, 0] = 0
        u, v = _curl(torch.fft.ifft2(hat).real, h)
        if flow == "turbulence":
            s = 1.0 / math.sqrt(0.5 * float((u * u + v * v).mean()))
            u, v = u * s, v * s
    umax = max(float(u.abs().max()), float(v.abs().max()))
    return u.float(), v.float(), 0.5 * h / umax


def _disks(c, seed):
    rng = np.random.default_rng([seed, 1])
    ly = TWO_PI / c["nx"] * c["ny"]
    short, found = min(TWO_PI, ly), []
    while len(found) < c["disks"]:
        r = float(rng.uniform(0.02, 0.08)) * short
        x, y = float(rng.uniform(0.15, 0.7)) * TWO_PI, float(rng.uniform(0.2, 0.8)) * ly
        if all(math.hypot(x - a, y - b) > r + q + 0.02 * short for a, b, q in found):
            found.append((x, y, r))
    return found


def _modes(c, seed):
    rng = np.random.default_rng([seed, 2])
    return [(int(rng.integers(2, 9)), int(rng.integers(-8, 9)), float(rng.uniform(0, TWO_PI))) for _ in range(c["modes"])]


def _pinned(*shape):
    return torch.empty(*shape, dtype=torch.float32, pin_memory=DEV == "cuda")


def _pin(t):
    return _pinned(*t.shape).copy_(t)


BAND = dict(kf=9.0, width=1.0, amplitude=3.0, drag=0.1)
FORCING = dict(amplitude=0.5, drag=0.1, phase_drift=0.3)
SIDES = (64, 128, 192, 256, 384, 512)


def _guess_inputs(case, seed):
    """normalised divergence with edges of disks in it, their mask, and the pressure that solves it"""
    B, H, W = case["batch"], case["h"], case["w"]
    rng = np.random.default_rng(seed)
    div = 0.2 * torch.randn(B, H, W, device=DEV, generator=_generator(seed))
    mask = torch.zeros(B, H, W, device=DEV)
    x, y = torch.arange(W, device=DEV)[None, :], torch.arange(H, device=DEV)[:, None]
    for b in range(B):
        for _ in range(int(rng.integers(1, 9))):
            r = float(rng.uniform(0.02, 0.08)) * H + 2
            d = torch.hypot(x - float(rng.uniform(0, W)), y - float(rng.uniform(0, H))) - r
            mask[b] = torch.maximum(mask[b], 0.5 * (1 - torch.tanh(d / 0.75)))
            div[b] += 3 * float(rng.normal()) * torch.exp(-(d / 1.5) ** 2)
    div -= div.mean((1, 2), keepdim=True)
    div /= div.square().mean((1, 2), keepdim=True).sqrt()
    ev = (2 * torch.cos(TWO_PI * torch.fft.fftfreq(W, device=DEV, dtype=torch.float64)) - 2)[None, :] + \
         (2 * torch.cos(TWO_PI * torch.fft.fftfreq(H, device=DEV, dtype=torch.float64)) - 2)[:, None]
    ev[0, 0] = 1
    hat = torch.fft.fft2(div.double()) / ev
    hat[:, 0, 0] = 0
    return div.contiguous(), mask.contiguous(), torch.fft.ifft2(hat).real.float().contiguous()


# ------------------------------------------------------------ prepare / run
def prepare(case, seed):
    c = case
    if c["kind"] in ("predict", "grad"):
        g = fs.PressureGuess(seed=0)
        g.load(WEIGHTS)
        g.set_loss(0.05, 1.0)
        div, mask, p = _guess_inputs(c, seed)
        return dict(kind=c["kind"], g=g, div=div, mask=mask, p=p)
    if c["kind"] == "batch":
        rng = np.random.default_rng(7)
        sides = [int(rng.choice(SIDES)) for _ in range(c["count"])]
        opts = dict(nu=1e-4, tol=1e-6)
        b = fs.GPUFluidBatch([dict(n=n, nu=opts["nu"], advection="maccormack", pressure_solver="multigrid",
                                   pressure_iterations=1, precision="mixed", pressure_tol=opts["tol"], max_cycles=60,
                                   relax=1.2) for n in sides])
        dts = []
        for i, n in enumerate(sides):
            u, v, dt = _flow(dict(nx=n, ny=n), seed * 1000 + i, "blobs")
            b.members[i].upload_velocity(u.cpu().numpy(), v.cpu().numpy())
            dts.append(dt)
        total = sum(n * n for n in sides)
        return dict(kind="batch", b=b, sides=sides, dts=dts, steps=c["steps"], u=_pinned(total), v=_pinned(total))
    if c["kind"] == "frame":
        c = dict(c, ny=c["nx"])
        u, v, dt = _flow(c, seed, "blobs")
        s = fs.GPUFluidSolver(n=c["nx"], pressure_solver="multigrid", pressure_iterations=c["iterations"],
                              dye_fade=0.002)
        dye = torch.rand(c["nx"], c["nx"], 4, device=DEV, generator=_generator(seed))
        img, out = _pinned(c["nx"], c["nx"], 4), _pinned(c["nx"], c["nx"], 4)
        return dict(kind="frame", s=s, u0=_pin(u), v0=_pin(v), dye=_pin(dye), dt=dt, frames=c["frames"], img=img, out=out)
    extra = dict(mg_first_pre=c["first"], mg_first_post=c["first"], pressure_tol_relative=c["relative"])
    ly = TWO_PI / c["nx"] * c["ny"]
    s = fs.GPUFluidSolver(nx=c["nx"], ny=c["ny"], lx=TWO_PI, ly=ly, nu=c["nu"], advection=c["advection"],
                          pressure_solver=c["pressure"], pressure_iterations=c["iterations"], precision=c["precision"],
                          pressure_tol=c["tol"], max_cycles=60, mg_coarse_sweeps=c["coarse"], relax=c["relax"], **extra)
    u, v, dt = _flow(c, seed)
    if c["modes"]:
        s.set_forcing(_modes(c, seed), **FORCING)
    if c["band"]:
        s.set_band_forcing("gaussian", seed=int(seed), **BAND)
    if c["channel"]:
        s.set_channel(fs.workload.channel_geometry())
    if c["disks"]:
        s.set_solids(_disks(c, seed))
    return dict(kind="steps", s=s, u0=_pin(u), v0=_pin(v), u=_pinned(c["ny"], c["nx"]), v=_pinned(c["ny"], c["nx"]),
                dt=dt, steps=c["steps"])


def run(state):
    st = state
    if st["kind"] == "predict":
        return st["g"].predict(st["div"], st["mask"])
    if st["kind"] == "grad":
        return st["g"].loss_grad(st["div"], st["mask"], st["p"])
    lib, check = fs.load(), fs._lib.check
    if st["kind"] == "batch":  # the simulations go on from pass to pass
        for _ in range(st["steps"]):
            st["b"].step(st["dts"])
        at = 0
        for m, n in zip(st["b"].members, st["sides"]):
            check(lib.fs_read_velocity(m._h, st["u"].data_ptr() + 4 * at, st["v"].data_ptr() + 4 * at, 0), m._h)
            at += n * n
        return st["u"], st["v"]
    s = st["s"]
    check(lib.fs_upload_velocity(s._h, st["u0"].data_ptr(), st["v0"].data_ptr(), 0), s._h)
    if st["kind"] == "frame":
        check(lib.fs_upload_dye(s._h, st["dye"].data_ptr()), s._h)
        for _ in range(st["frames"]):
            s.step(st["dt"])
            check(lib.fs_render(s._h, 0, 0.5, st["img"].data_ptr()), s._h)
        check(lib.fs_read_dye(s._h, st["out"].data_ptr()), s._h)
        return st["img"], st["out"]
    s.advance(st["dt"], st["steps"])
    check(lib.fs_read_velocity(s._h, st["u"].data_ptr(), st["v"].data_ptr(), 0), s._h)
    return st["u"], st["v"]


# --------------------------------------------------------------------- work
def _step_work(cells, mixed, mc, pressure, iterations, tol):
    """bytes and operations of one step: the state read and written once; ~100 operations per cell for an advection
    pass, 8 per sweep, ~60 per V(2,2) cycle over all levels"""
    cycles = iterations if not tol else (5 if tol >= 1e-6 else 8)
    solve = 60 * cycles if pressure == "multigrid" else 8 * iterations * (2 if pressure == "red-black" else 1)
    return cells * (32 if mixed else 16), cells * ((200 if mc else 100) + 30 + solve)


CONVS = ((2, 16, 1), (16, 16, 1), (16, 32, 4), (32, 64, 16), (64, 128, 64), (128, 64, 64), (64, 32, 16), (32, 16, 4),
         (16, 16, 1), (16, 1, 1))  # channels in, out, and the cells one cell of this level stands for


def work(case):
    c = case
    if c["kind"] in ("predict", "grad"):
        px = c["batch"] * c["h"] * c["w"]
        flops = sum(18 * ci * co / area for ci, co, area in CONVS) * px
        return dict(bytes=px * (12 if c["kind"] == "predict" else 16), flops=flops * (1 if c["kind"] == "predict" else 3))
    if c["kind"] == "batch":
        rng = np.random.default_rng(7)
        cells = sum(int(rng.choice(SIDES)) ** 2 for _ in range(c["count"]))
        b, f = _step_work(cells, True, True, "multigrid", 1, 1e-6)
        return dict(bytes=b * c["steps"], flops=f * c["steps"])
    if c["kind"] == "frame":
        cells = c["nx"] ** 2
        b, f = _step_work(cells, False, True, "multigrid", c["iterations"], 0)
        return dict(bytes=(b + 48 * cells) * c["frames"], flops=(f + 150 * cells) * c["frames"])
    b, f = _step_work(c["nx"] * c["ny"], c["precision"] == "mixed", c["advection"] == "maccormack", c["pressure"],
                      c["iterations"], c["tol"])
    return dict(bytes=b * c["steps"], flops=f * c["steps"])


# -------------------------------------------------- the same in 64 bits
def _corner_values(f, x, y):
    """the four values around index-space points (x, y) of a periodic field, and the weights"""
    ny, nx = f.shape[:2]
    i, j = torch.floor(x), torch.floor(y)
    fx, fy = x - i, y - j
    i0, j0 = i.long() % nx, j.long() % ny
    i1, j1 = (i0 + 1) % nx, (j0 + 1) % ny
    return f[j0, i0], f[j0, i1], f[j1, i0], f[j1, i1], fx, fy


def _sample(f, x, y):
    a, b, c, d, fx, fy = _corner_values(f, x, y)
    if f.dim() == 3:
        fx, fy = fx[..., None], fy[..., None]
    top, bot = a + (b - a) * fx, c + (d - c) * fx
    return top + (bot - top) * fy


def _depart(u, v, px, py, cx, cy):
    """RK2 backward trace of points (in cells; u at (i, j+1/2), v at (i+1/2, j))"""
    mx = px - 0.5 * cx * _sample(u, px, py - 0.5)
    my = py - 0.5 * cy * _sample(v, px - 0.5, py)
    return px - cx * _sample(u, mx, my - 0.5), py - cy * _sample(v, mx - 0.5, my)


def _advect(u, v, cx, cy, maccormack):
    ny, nx = u.shape
    I = torch.arange(nx, device=u.device, dtype=torch.float64).expand(ny, nx)
    J = torch.arange(ny, device=u.device, dtype=torch.float64)[:, None].expand(ny, nx)
    homes = ((I, J + 0.5, 0.0, 0.5), (I + 0.5, J, 0.5, 0.0))
    fwd, lo, hi = [], [], []
    for f, (px, py, ox, oy) in zip((u, v), homes):
        x, y = _depart(u, v, px, py, cx, cy)
        a, b, c, d, _, _ = _corner_values(f, x - ox, y - oy)
        fwd.append(_sample(f, x - ox, y - oy))
        lo.append(torch.minimum(torch.minimum(a, b), torch.minimum(c, d)))
        hi.append(torch.maximum(torch.maximum(a, b), torch.maximum(c, d)))
    if not maccormack:
        return fwd
    out = []
    for f, g, l, m, (px, py, ox, oy) in zip((u, v), fwd, lo, hi, homes):
        x, y = _depart(u, v, px, py, -cx, -cy)
        out.append(torch.minimum(torch.maximum(g + 0.5 * (f - _sample(g, x - ox, y - oy)), l), m))
    return out


def _nb(p):
    return torch.roll(p, 1, 1) + torch.roll(p, -1, 1) + torch.roll(p, 1, 0) + torch.roll(p, -1, 0)


def _rb(p, d, h2, sweeps):
    ny, nx = p.shape
    red = ((torch.arange(nx, device=p.device)[None, :] + torch.arange(ny, device=p.device)[:, None]) % 2) == 0
    for _ in range(sweeps):
        for colour in (red, ~red):
            p = torch.where(colour, (_nb(p) - h2 * d) / 4, p)
    return p


def _vcycle(p, d, h2):
    n = p.shape[0]
    if n // 2 < 8 or n % 2:
        return _rb(p, d, h2, 40)
    p = _rb(p, d, h2, 2)
    r = d - (_nb(p) - 4 * p) / h2
    rc = r.reshape(n // 2, 2, n // 2, 2).mean((1, 3))
    e = _vcycle(torch.zeros_like(rc), rc, 4 * h2)
    for dim in (0, 1):  # bilinear: 3/4 of the own coarse cell, 1/4 of the neighbour
        lo, hi = 0.75 * e + 0.25 * torch.roll(e, 1, dim), 0.75 * e + 0.25 * torch.roll(e, -1, dim)
        e = torch.stack((lo, hi), dim + 1).flatten(dim, dim + 1)
    return _rb(p + e, d, h2, 2)


def _project(u, v, h, pressure, iterations, tol):
    d = (torch.roll(u, -1, 1) - u + torch.roll(v, -1, 0) - v) / h
    ny, nx = d.shape
    p = torch.zeros_like(d)
    if tol:  # to a tolerance: the exact solution
        ev = (2 * torch.cos(TWO_PI * torch.arange(nx, device=d.device, dtype=torch.float64) / nx) - 2)[None, :] + \
             (2 * torch.cos(TWO_PI * torch.arange(ny, device=d.device, dtype=torch.float64) / ny) - 2)[:, None]
        ev[0, 0] = 1
        hat = torch.fft.fft2(d) * h * h / ev
        hat[0, 0] = 0
        p = torch.fft.ifft2(hat).real
    elif pressure == "jacobi":
        for _ in range(iterations):
            p = (_nb(p) - h * h * d) / 4
    elif pressure == "red-black":
        p = _rb(p, d, h * h, iterations)
    else:
        for _ in range(iterations):
            p = _vcycle(p, d, h * h)
    return u - (p - torch.roll(p, 1, 1)) / h, v - (p - torch.roll(p, 1, 0)) / h


def _faces(nx, ny, h):
    i = torch.arange(nx, device=DEV, dtype=torch.float64)[None, :] * h
    j = torch.arange(ny, device=DEV, dtype=torch.float64)[:, None] * h
    return (i, j + 0.5 * h), (i + 0.5 * h, j)


def _toward(f, chi, target):
    return torch.where(chi >= 1e-6, f + chi * (target - f), f)


def _wrapped(d, L):
    return d - L * torch.floor(d / L + 0.5)


def _solids(u, v, h, ly, disks, channel):
    faces = _faces(u.shape[1], u.shape[0], h)
    out = []
    for f, (x, y), inflow in ((u, faces[0], 1.0), (v, faces[1], 0.0)):
        if channel:
            g = channel
            chi = 0.5 * (1 - torch.tanh((_wrapped(x - g["fringe_x"], TWO_PI).abs() - g["fringe_half"]) / g["fringe_ramp"]))
            f = _toward(f, chi.expand_as(f), inflow * g["inflow_u"])
            chi = 0.5 * (1 - torch.tanh((_wrapped(y - g["wall_y"], ly).abs() - g["wall_half"]) / (1.5 * h)))
            f = _toward(f, chi.expand_as(f), 0.0)
        for a, b, r in disks:
            dist = torch.hypot(_wrapped(x - a, TWO_PI), _wrapped(y - b, ly))
            f = _toward(f, 0.5 * (1 - torch.tanh((dist - r) / (1.5 * h))), 0.0)
        out.append(f)
    return out


def _forcing(u, v, h, dt, t, modes):
    (xu, yu), (xv, yv) = _faces(u.shape[1], u.shape[0], h)
    fu, fv = torch.zeros_like(u), torch.zeros_like(v)
    for kx, ky, ph in modes:
        kk, ph = math.hypot(kx, ky), ph + FORCING["phase_drift"] * t
        fu += ky / kk * torch.cos(kx * xu + ky * yu + ph)
        fv -= kx / kk * torch.cos(kx * xv + ky * yv + ph)
    scale, damp = FORCING["amplitude"] * dt / math.sqrt(len(modes)), math.exp(-FORCING["drag"] * dt)
    return u * damp + scale * fu, v * damp + scale * fv


def _philox(step, modes, key):
    """Philox4x32-10 (Salmon et al., SC'11): the first two words of counters (step, mode, 0, 0)"""
    M32 = np.uint64(0xFFFFFFFF)
    x = [np.full(modes, step, np.uint64), np.arange(modes, dtype=np.uint64), np.zeros(modes, np.uint64), np.zeros(modes, np.uint64)]
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * x[0], np.uint64(0xCD9E8D57) * x[2]
        x = [(b >> np.uint64(32)) ^ x[1] ^ np.uint64(k0), b & M32, (a >> np.uint64(32)) ^ x[3] ^ np.uint64(k1), a & M32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return x[0].astype(np.float64), x[1].astype(np.float64)


def _band_forcing(u, v, h, dt, step, seed):
    lo, hi = BAND["kf"] - BAND["width"], BAND["kf"] + BAND["width"]
    K = math.ceil(hi)
    lattice = [(kx, ky) for ky in range(-K, K + 1) for kx in range(-K, K + 1) if lo * lo <= kx * kx + ky * ky <= hi * hi]
    r0, r1 = _philox(step, len(lattice), int(seed))
    A, phi = np.sqrt(-2 * np.log((r0 + 0.5) / 2**32)), TWO_PI * (r1 + 0.5) / 2**32
    (xu, yu), (xv, yv) = _faces(u.shape[1], u.shape[0], h)
    s = BAND["amplitude"] * dt / math.sqrt(len(lattice))
    for (kx, ky), a, p in zip(lattice, A, phi):
        kk = math.hypot(kx, ky)
        u = u + s * a * ky / kk * torch.cos(kx * xu + ky * yu + p)
        v = v - s * a * kx / kk * torch.cos(kx * xv + ky * yv + p)
    damp = math.exp(-BAND["drag"] * dt)
    return u * damp, v * damp


def _steps64(c, seed, u, v, dt, steps):
    h = TWO_PI / c["nx"]
    ly = h * c["ny"]
    u, v = u.double(), v.double()
    modes, disks = _modes(c, seed), _disks(c, seed)
    channel = fs.workload.channel_geometry() if c["channel"] else None
    for k in range(steps):
        u, v = _advect(u, v, dt / h, dt / h, c["advection"] == "maccormack")
        if c["nu"]:
            a = c["nu"] * dt / (h * h)
            u, v = u + a * (_nb(u) - 4 * u), v + a * (_nb(v) - 4 * v)
        if c["band"]:
            u, v = _band_forcing(u, v, h, dt, k, seed)
        if modes:
            u, v = _forcing(u, v, h, dt, k * dt, modes)
        if channel or disks:
            u, v = _solids(u, v, h, ly, disks, channel)
        u, v = _project(u, v, h, c["pressure"], c["iterations"], c["tol"])
    return u, v


def _ramp(e0, e1, x):
    t = ((x - e0) / (e1 - e0)).clamp(0, 1)
    return t * t * (3 - 2 * t)


def _image(u, v, dye, h, exposure):
    """the vorticity rendering in 64 bits"""
    w = (v - torch.roll(v, 1, 1) - u + torch.roll(u, 1, 0)) / h
    w = w + torch.roll(w, -1, 1)
    w = 0.25 * (w + torch.roll(w, -1, 0))
    speed = torch.hypot(u, v)
    rgb = lambda *t: torch.tensor(t, device=u.device, dtype=torch.float64)  # noqa: E731
    sig = torch.tanh((w * exposure).clamp(-12, 12))[..., None]
    mag = sig.abs()
    hue = torch.where(sig >= 0, rgb(1.00, 0.10, 0.62), rgb(0.10, 0.92, 1.00))
    col = torch.lerp(rgb(0.004, 0.003, 0.016).expand_as(hue), rgb(0.16, 0.03, 0.42).expand_as(hue), _ramp(0, 0.22, mag))
    col = torch.lerp(col, hue, _ramp(0.12, 0.62, mag)) * (0.30 + 4.6 * mag * mag)
    sp = torch.tanh((speed * exposure * 0.45).clamp(0, 12))[..., None]
    col = col + rgb(0.55, 0.78, 1.0) * sp ** 5 * 0.85
    lum = (dye[..., :3] * rgb(0.2126, 0.7152, 0.0722)).sum(-1, keepdim=True)
    col = col + col * lum * 1.5 + dye[..., :3] * 0.20
    return torch.cat((col, torch.ones_like(lum)), -1)


def _frames64(case, seed):
    n = case["nx"]
    h = TWO_PI / n
    u, v, dt = _flow(dict(nx=n, ny=n), seed, "blobs")
    dye = torch.rand(n, n, 4, device=DEV, generator=_generator(seed)).double()
    c = steps_case(nx=n, ny=n, pressure="multigrid", iterations=case["iterations"])
    I = torch.arange(n, device=DEV, dtype=torch.float64) + 0.5
    X, Y = I.expand(n, n), I[:, None].expand(n, n)
    for _ in range(case["frames"]):
        u, v = _steps64(c, seed, u, v, dt, 1)
        x, y = _depart(u, v, X, Y, dt / h, dt / h)
        dye = (_sample(dye, x - 0.5, y - 0.5) * (1 - 0.002)).clamp(0, 1)
    return _image(u, v, dye, h, 0.5), dye


NET = ((16, 16), (16, 16), (16, 32), (32, 64), (64, 128), (128, 64), (64, 32), (32, 16), (16, 16), (16, 16))


def _network64(theta, div, mask):
    F = torch.nn.functional
    at, layers = 0, []
    for ci, co in NET:
        w = theta[at:at + co * ci * 9].view(co, ci, 3, 3)
        b = theta[at + co * ci * 9:at + co * ci * 9 + co]
        at += co * (ci * 9 + 1)
        layers.append((w, b))

    def conv(x, k):
        w, b = layers[k]
        return F.conv2d(F.pad(x, (1, 1, 1, 1), mode="circular"), w[:, :x.shape[1]], b)

    up = lambda x: x.repeat_interleave(2, 2).repeat_interleave(2, 3)  # noqa: E731
    pool = lambda x: F.avg_pool2d(x, 2)  # noqa: E731
    a0 = conv(conv(torch.stack((div, mask), 1).double(), 0).relu(), 1).relu()
    a1 = conv(pool(a0), 2).relu()
    a2 = conv(pool(a1), 3).relu()
    f3 = conv(conv(pool(a2), 4).relu(), 5).relu()
    g2 = conv(up(f3) + a2, 6).relu()
    h1 = conv(up(g2) + a1, 7).relu()
    return conv(conv(up(h1) + a0, 8).relu(), 9)[:, 0]


def exact(case, seed):
    c = case
    if c["kind"] == "steps":
        u, v, dt = _flow(c, seed)
        return _steps64(c, seed, u, v, dt, c["steps"])
    if c["kind"] == "frame":
        return _frames64(c, seed)
    if c["kind"] == "batch":
        rng = np.random.default_rng(7)
        us, vs = [], []
        for i in range(c["count"]):
            n = int(rng.choice(SIDES))
            u, v, dt = _flow(dict(nx=n, ny=n), seed * 1000 + i, "blobs")
            u, v = _steps64(steps_case(nx=n, ny=n, nu=1e-4, tol=1e-6, **MIXED), seed, u, v, dt, c["steps"])
            us.append(u.reshape(-1))
            vs.append(v.reshape(-1))
        return torch.cat(us), torch.cat(vs)
    div, mask, p = _guess_inputs(c, seed)
    theta = torch.from_numpy(np.fromfile(WEIGHTS, "<f4", offset=16).astype(np.float64)).to(DEV)
    if c["kind"] == "predict":
        with torch.no_grad():
            return _network64(theta, div, mask)
    theta.requires_grad_(True)
    e = _network64(theta, div, mask) - p.double()
    lap = torch.roll(e, 1, 1) + torch.roll(e, -1, 1) + torch.roll(e, 1, 2) + torch.roll(e, -1, 2) - 4 * e
    loss = 0.05 * (e - e.mean((1, 2), keepdim=True)).square().mean() + lap.square().mean()
    (grad,) = torch.autograd.grad(loss, theta)
    return float(loss), grad
