"""The work a user has this library do, as cases whose speed and results can be measured.

Every case is a call, or a few calls in the order in which a simulation makes them, through
the public entry points (the Python binding and the C ABI in include/pic_gb300.h). Grids
have unit cells; sizes, densities and time steps are those of the benchmark configurations
and of the tests, and a few odd ones.

Inputs are made with torch on the GPU from the seed alone and uploaded as a user's program
uploads its FP64 particle arrays. Results that come back to the host arrive in page-locked
buffers (pic_gpu_host_alloc's kind), except in the host-array calls, which return what the
mirror of the reference's interface returns.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

NGP, CIC, TSC, ESK = 0, 1, 2, 3
SCHEMES = {"NGP": NGP, "CIC": CIC, "TSC": TSC, "ESK": ESK}
DEP_FLOPS = {"NGP": 6, "CIC": 15, "TSC": 45, "ESK": 40}  # per particle, weights and sums
NET = [(16, 32), (32, 32), (32, 32), (32, 32), (32, 32), (32, 16)]  # channels of the network's layers


def _binding():
    path = os.path.join(ROOT, "pic-deposition_gb300")
    if path not in sys.path:
        sys.path.insert(0, path)
    import pic_gb300

    return pic_gb300


def listed():
    return [
        # The drop-in call of the reference's interface on a test-sized problem: host arrays
        # in, rho out. Latency and the number of launches and copies count.
        dict(name="call_cic_64", kind="call", nx=64, ny=64, ppc=16, scheme="CIC", sorted=False, vth=0.0, dt=0.0),
        # The same call at the reference's own benchmark size: 1,048,576 particles, uniform.
        dict(name="call_cic_256", kind="call", nx=256, ny=256, ppc=16, scheme="CIC", sorted=False, vth=0.0, dt=0.0),
        # The headline workload: CIC charge of 67,108,864 cell-sorted resident particles.
        dict(name="deposit_cic_1024", kind="deposit", nx=1024, ny=1024, ppc=64, scheme="CIC", order="sorted",
             species=1, amp=0.01, vth=0.1, dt=0.1),
        # Two species (per-particle charges) on a grid that no tile divides, the smoothest shape.
        dict(name="deposit_tsc_odd", kind="deposit", nx=777, ny=513, ppc=40, scheme="TSC", order="sorted", species=2,
             amp=0.05, vth=0.1, dt=0.1),
        # The Esirkepov workload: trajectory charge and the charge-conserving current of one move.
        dict(name="esirkepov_1024", kind="esirkepov", nx=1024, ny=1024, ppc=64, species=1, amp=0.01, vth=0.1, dt=0.1),
        # A cell sort after ten steps' drift, with the permutation for the user's own arrays.
        dict(name="sort_1024", kind="sort", nx=1024, ny=1024, ppc=16, species=1, amp=0.01, vth=0.1, dt=1.0),
        # The time step at the size of the reference's validation runs: bound by launches.
        dict(name="step_cic_64", kind="step", nx=64, ny=64, ppc=16, scheme="CIC", v0=0.0, vth=0.05, amp=0.01, dt=0.1,
             steps=100, sort_interval=20, particles=True),
        # The Landau set-up of the warm-start study: a hot plasma whose particles leave their
        # cells between sorts.
        dict(name="step_cic_512", kind="step", nx=512, ny=512, ppc=64, scheme="CIC", v0=0.0, vth=1.0, amp=0.05, dt=0.1,
             steps=20, sort_interval=10, particles=True),
        # The two-stream production run (TSC, 100 per cell, sort every ten steps): the largest.
        dict(name="step_tsc_1024", kind="step", nx=1024, ny=1024, ppc=100, scheme="TSC", v0=0.2, vth=0.01, amp=0.0,
             dt=0.1, steps=10, sort_interval=10, particles=False),
        # A red-black Gauss-Seidel Poisson solve from zero to the study's tolerance.
        dict(name="rbgs_256", kind="rbgs", nx=256, ny=256, tol=1e-8, mixed=False),
        # A batch of independent Langmuir runs of uneven size, a stretch of its 500 steps.
        dict(name="ensemble_8", kind="ensemble", members="128x4,128x16,128x64,128x256,256x16,256x64,512x4,512x16",
             steps=100, sort_interval=20),
        # One loss and gradient of the warm-start network at the study's batch: forward and
        # backward through all its layers.
        dict(name="network_512", kind="network", nx=512, ny=512, batch=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "deposit", "deposit", "esirkepov", "sort", "step", "step", "rbgs", "ensemble", "network"])
    if kind == "rbgs":
        return dict(kind=kind, nx=2 * _log(rng, 16, 112), ny=2 * _log(rng, 16, 112), tol=rng.choice([1e-6, 1e-8]),
                    mixed=rng.random() < 0.5)
    if kind == "ensemble":
        members = ["%dx%d" % (rng.choice([64, 128, 256]), rng.choice([4, 16, 64])) for _ in range(rng.randint(2, 8))]
        return dict(kind=kind, members=",".join(members), steps=rng.randint(40, 90), sort_interval=rng.choice([10, 20]))
    if kind == "network":
        return dict(kind=kind, nx=128 * rng.randint(1, 4), ny=2 * _log(rng, 32, 256), batch=rng.randint(1, 15))
    top = 512 if kind == "call" else 1500 if kind == "deposit" else 1024
    most = 4e6 if kind == "call" else 6e7 if kind != "step" else 3e7
    nx, ny = _log(rng, 24, top), _log(rng, 24, top)
    ppc = _log(rng, 2, max(2.0, min(128.0, most / (nx * ny))))
    scheme = rng.choice(["NGP", "CIC", "TSC", "ESK"])
    case = dict(kind=kind, nx=nx, ny=ny, ppc=ppc)
    if kind == "call":
        return dict(case, scheme=scheme, sorted=rng.random() < 0.5, vth=0.1, dt=0.1)
    if kind == "step":
        return dict(case, scheme=scheme, v0=rng.choice([0.0, 0.2]), vth=rng.choice([0.01, 0.05, 1.0]),
                    amp=rng.choice([0.0, 0.01, 0.05]), dt=0.1, steps=rng.randint(10, 40),
                    sort_interval=rng.choice([1, 5, 10, 20]), particles=True)
    case.update(species=rng.choice([1, 1, 2]), amp=rng.choice([0.0, 0.01, 0.05]), vth=rng.choice([0.1, 1.0]), dt=0.1)
    if kind == "deposit":
        case.update(scheme=scheme, order=rng.choice(["sorted", "sorted", "random"]))
    elif kind == "sort":
        case.update(dt=rng.choice([0.1, 1.0]))
    return case


# ---- inputs -----------------------------------------------------------------------------


def _device():
    return torch.device("cuda")


def _rand(seed):
    return torch.Generator(device=_device()).manual_seed(seed)


def _particles(case, seed):
    """FP64 particle arrays on the GPU: x from the density 1 + amp cos(2 pi x / nx) (inverse of
    its distribution function by Newton steps), y uniform, Maxwellian velocities and two beams
    when v0 is given; charge -1, or -1/N in a time step, or two species of -1 and +2."""
    g = _rand(seed)
    nx, ny = case["nx"], case["ny"]
    n = nx * ny * case["ppc"]
    kw = dict(device=_device(), dtype=torch.float64, generator=g)
    x = torch.rand(n, **kw) * nx
    amp = case.get("amp", 0.0)
    if amp:
        k = 2.0 * math.pi / nx
        u = x.clone()
        for _ in range(5):
            x -= (x + (amp / k) * torch.sin(k * x) - u) / (1.0 + amp * torch.cos(k * x))
        x.clamp_(0.0, nx * (1.0 - 1e-12))
    y = torch.rand(n, **kw) * ny
    vth, v0 = case.get("vth", 0.0), case.get("v0", 0.0)
    vx = torch.randn(n, **kw) * vth
    vy = torch.randn(n, **kw) * vth
    if v0:
        vx[: n // 2] += v0
        vx[n // 2:] -= v0
    if case["kind"] == "step":
        q = torch.full((n,), -1.0 / n, device=_device(), dtype=torch.float64)
    elif case.get("species", 1) == 2:
        q = torch.where(torch.rand(n, **kw) < 0.5, -1.0, 2.0)
    else:
        q = torch.full((n,), -1.0, device=_device(), dtype=torch.float64)
    return dict(x=x, y=y, vx=vx, vy=vy, q=q)


_stage = {}  # page-locked upload buffers, one per field, reused by every case


def _upload(ctx, p):
    host = {}
    for k, v in p.items():
        if k not in _stage or _stage[k].numel() < v.numel():
            _stage[k] = torch.empty(v.numel(), dtype=torch.float64, pin_memory=True)
        host[k] = _stage[k][: v.numel()]
        host[k].copy_(v)
    torch.cuda.synchronize()
    ctx.upload(host["x"].numpy(), host["y"].numpy(), host["q"].numpy(), host["vx"].numpy(), host["vy"].numpy())
    ctx._keep = None


def _pinned(n, dtype=torch.float64):
    return torch.empty(n, dtype=dtype, pin_memory=True)


def _network_params(seed):
    """He-normal weights w[tap][cout][cin] and small biases, zero in the unused channels."""
    g = torch.Generator().manual_seed(seed)
    parts = []
    for l, (ci, co) in enumerate(NET):
        cu, ou = (1 if l == 0 else ci), (1 if l == len(NET) - 1 else co)
        w = torch.zeros(9, co, ci)
        w[:, :ou, :cu] = torch.randn(9, ou, cu, generator=g) * math.sqrt(2.0 / (9.0 * cu))
        b = torch.zeros(co)
        b[:ou] = torch.randn(ou, generator=g) * 0.02
        parts += [w.reshape(-1), b]
    return torch.cat(parts)


def _network_fields(case, seed):
    g = _rand(seed)
    shape = (case["batch"], case["ny"], case["nx"])
    inp = torch.randn(shape, device=_device(), generator=g)
    tgt = torch.randn(shape, device=_device(), generator=g) * 0.3
    # values that BF16 holds, as the study's stored pairs are
    return inp.bfloat16().float(), tgt.bfloat16().float()


def _rbgs_rho(case, seed):
    """A perturbed density with the shot noise of 64 particles per cell."""
    nx, ny = case["nx"], case["ny"]
    g = _rand(seed)
    x = torch.arange(nx, device=_device(), dtype=torch.float64)
    rho = 1.0 + 0.05 * torch.cos(2.0 * math.pi * x / nx)[None, :].expand(ny, nx)
    return (rho + 0.125 * torch.randn((ny, nx), device=_device(), dtype=torch.float64, generator=g)).contiguous()


def prepare(case, seed):
    pg = _binding()
    kind = case["kind"]
    s = dict(case=case, pg=pg, lib=pg.lib())
    if kind == "ensemble":
        runs = [tuple(int(v) for v in m.split("x")) for m in case["members"].split(",")]
        s["ens"] = pg.Ensemble([(n, p, 100 * seed + i) for i, (n, p) in enumerate(runs)], dt=0.1, amplitude=0.01,
                               vth=0.05, sort_interval=case["sort_interval"], use_graph=True, seed=1)
        sizes = [s["ens"].info(i)["N"] ** 2 for i in range(len(runs))]
        s["rho"], s["phi"] = [_pinned(g) for g in sizes], [_pinned(g) for g in sizes]
        return s
    nx, ny = case["nx"], case["ny"]
    G = nx * ny
    if kind == "call":
        p = _particles(case, seed)
        soa = pg.ParticlesSoA(len(p["x"]))
        for k, v in p.items():
            setattr(soa, k, v.cpu().numpy())
        s["soa"], s["grid"] = soa, pg.FieldGrid(pg.Domain(float(nx), float(ny), nx, ny))
        s["config"] = pg.DepositionConfig(scheme=pg.DepositionScheme(SCHEMES[case["scheme"]]), sorted=case["sorted"],
                                          esirkepov_dt=case["dt"])
        return s
    if kind == "network":
        s["ctx"] = pg.Context(nx, ny, float(nx), float(ny), 16)
        s["ctx"].ws_init(seed=1)
        s["ctx"].ws_set_params(_network_params(seed).numpy())
        s["inputs"], s["targets"] = (t.cpu().pin_memory().numpy() for t in _network_fields(case, seed))
        return s
    if kind == "rbgs":
        s["ctx"] = pg.Context(nx, ny, float(nx), float(ny), 16)
        s["ctx"].set_rho(_rbgs_rho(case, seed).cpu().numpy().reshape(-1))
        s["ctx"].set_rbgs_precision(case["mixed"])
        s["out"] = [_pinned(G) for _ in range(3)]
        return s
    p = _particles(case, seed)
    n = len(p["x"])
    s["n"] = n
    s["ctx"] = pg.Context(nx, ny, float(nx), float(ny), n)
    _upload(s["ctx"], p)
    if kind == "esirkepov" or (kind == "deposit" and case["order"] == "sorted"):
        s["ctx"].sort()
    if kind == "deposit":
        s["out"] = [_pinned(G)]
    elif kind == "esirkepov":
        s["out"] = [_pinned(G) for _ in range(3)]
    elif kind == "sort":
        s["out"] = [_pinned(n, torch.int32), _pinned(G + 1, torch.int32)]
    else:
        s["out"] = [_pinned(G) for _ in range(4)]
        if case["particles"]:
            s["out"] += [_pinned(n, torch.int32)] + [_pinned(n, torch.float32) for _ in range(4)]
    return s


# ---- the measured calls -------------------------------------------------------------------


def _ok(s, rc):
    if rc != 0:
        raise RuntimeError(s["lib"].pic_gpu_last_error().decode())


def run(s):
    case, lib = s["case"], s["lib"]
    kind = case["kind"]
    if kind == "call":
        s["pg"].depositChargeSoA(s["soa"], s["grid"], s["config"])
        return s["grid"].rho
    if kind == "ensemble":
        fe, ke = s["ens"].run(case["steps"])
        for i, (rho, phi) in enumerate(zip(s["rho"], s["phi"])):
            _ok(s, lib.pic_ens_download_run(s["ens"].h, i, None, None, None, None, rho.data_ptr(), phi.data_ptr()))
        return [fe, ke, s["rho"], s["phi"]]
    ctx = s["ctx"]
    if kind == "network":
        loss, grad = ctx.ws_loss_grad(s["inputs"], s["targets"])
        return [loss, grad]
    out = s["out"]
    ptr = [t.data_ptr() for t in out]
    if kind == "deposit":
        _ok(s, lib.pic_gpu_deposit(ctx.h, SCHEMES[case["scheme"]], case["dt"], 0.0, ptr[0]))
        return out
    if kind == "esirkepov":
        _ok(s, lib.pic_gpu_deposit(ctx.h, ESK, case["dt"], 0.0, ptr[0]))
        _ok(s, lib.pic_gpu_deposit_current(ctx.h, case["dt"], ptr[1], ptr[2]))
        return out
    if kind == "sort":
        ctx.push(case["dt"])
        _ok(s, lib.pic_gpu_sort(ctx.h, None, ptr[0], ptr[1]))
        return out
    if kind == "rbgs":
        iters, resid = ctx.poisson_rbgs(tol=case["tol"], max_iters=1000000, warm_start=False, check_every=64)
        _ok(s, lib.pic_gpu_get_fields(ctx.h, ptr[0], ptr[1], ptr[2]))
        return [iters, resid] + out
    history = ctx.run(case["steps"], scheme=SCHEMES[case["scheme"]], dt=case["dt"],
                      background=1.0 / (case["nx"] * case["ny"]), sort_interval=case["sort_interval"], use_graph=True)
    _ok(s, lib.pic_gpu_get_rho(ctx.h, ptr[0]))
    _ok(s, lib.pic_gpu_get_fields(ctx.h, ptr[1], ptr[2], ptr[3]))
    if case["particles"]:
        _ok(s, lib.pic_gpu_download_device_layout(ctx.h, *ptr[4:9], None))
    return [history] + out


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        runs = [tuple(int(v) for v in m.split("x")) for m in case["members"].split(",")]
        n, g = sum(a * a * p for a, p in runs), sum(a * a for a, p in runs)
        return {"bytes": case["steps"] * (40.0 * n + 32.0 * g), "flops": case["steps"] * (55.0 * n + 100.0 * g)}
    g = float(case["nx"] * case["ny"])
    if kind == "network":
        macs = 9.0 * (32 + 4 * 32 * 32 + 32)
        return {"bytes": 8.0 * g * case["batch"] + 8.0 * 40000, "flops": 6.0 * macs * g * case["batch"]}
    if kind == "rbgs":
        k = 2.0 * math.pi / max(case["nx"], case["ny"])
        return {"bytes": 32.0 * g, "flops": 7.0 * g * math.log(1.0 / case["tol"]) / (k * k)}
    n = g * case["ppc"]
    if kind == "call":
        esk = case["scheme"] == "ESK"
        return {"bytes": (40.0 if esk else 24.0) * n + 8.0 * g, "flops": DEP_FLOPS[case["scheme"]] * n}
    two = 4.0 if case.get("species", 1) == 2 else 0.0
    if kind == "deposit":
        per = 8.0 + two + (8.0 if case["scheme"] == "ESK" else 0.0) + (4.0 if case["order"] == "random" else 0.0)
        return {"bytes": per * n + 8.0 * g, "flops": DEP_FLOPS[case["scheme"]] * n}
    if kind == "esirkepov":
        return {"bytes": (16.0 + two) * n + 24.0 * g, "flops": (DEP_FLOPS["ESK"] + 90.0) * n}
    if kind == "sort":
        return {"bytes": (44.0 + 2.0 * two) * n + 4.0 * g, "flops": 6.0 * n}
    per = case["steps"] * (40.0 * n + 40.0 * g) + (20.0 * n if case["particles"] else 0.0)
    return {"bytes": per, "flops": case["steps"] * ((40.0 + DEP_FLOPS[case["scheme"]]) * n + 100.0 * g)}


# ---- the same results in 64 bits, by plain torch ------------------------------------------


def _axis(r, v, scheme, dt):
    """First node (relative to the particle's cell) and node weights of one axis."""
    one = torch.ones_like(r)
    if scheme == NGP:
        up = (r >= 0.5).double()
        return 0, [one - up, up]
    if scheme == CIC:
        return 0, [one - r, r]
    if scheme == TSC:
        up = r >= 0.5
        t = torch.where(up, r - 1.0, r)
        a, b, c = 0.5 * (0.5 - t) ** 2, 0.75 - t * t, 0.5 * (0.5 + t) ** 2
        z = torch.zeros_like(r)
        return -1, [torch.where(up, z, a), torch.where(up, a, b), torch.where(up, b, c), torch.where(up, c, z)]
    d = v * dt
    e = r + d
    still = d.abs() < 1e-15
    hi = torch.where(e > 1.0, (e - 1.0) / torch.where(still, one, e - r), 0.0 * r)
    lo = torch.where(e < 0.0, (0.0 - e) / torch.where(still, one, r - e), 0.0 * r)
    hi, lo = torch.where(still, r, hi), torch.where(still, 0.0 * r, lo)
    return -1, [lo, one - hi - lo, hi]


def _split(x, n):
    f = torch.floor(x)
    return f.long() % n, x - f


def _deposit64(p, nx, ny, scheme, dt):
    ix, rx = _split(p["x"], nx)
    iy, ry = _split(p["y"], ny)
    ax, wx = _axis(rx, p["vx"], scheme, dt)
    ay, wy = _axis(ry, p["vy"], scheme, dt)
    rho = torch.zeros(nx * ny, device=_device(), dtype=torch.float64)
    for j, b in enumerate(wy):
        for i, a in enumerate(wx):
            rho.index_add_(0, (iy + ay + j) % ny * nx + (ix + ax + i) % nx, p["q"] * b * a)
    return rho


def _current64(p, nx, ny, dt):
    """Esirkepov's first-order current of the move x -> x + v dt (moves below one cell)."""
    ix, rx = _split(p["x"], nx)
    iy, ry = _split(p["y"], ny)

    def shapes(r, d):
        zero = torch.zeros_like(r)
        s0 = [zero, 1.0 - r, r, zero]
        f = torch.floor(r + d)
        e = r + d - f
        k = f.long() + 1
        s1 = [torch.where(k == i, 1.0 - e, zero) + torch.where(k == i - 1, e, zero) for i in range(4)]
        return s0, [b - a for a, b in zip(s0, s1)]

    sx, dx = shapes(rx, p["vx"] * dt)
    sy, dy = shapes(ry, p["vy"] * dt)
    jx = torch.zeros(nx * ny, device=_device(), dtype=torch.float64)
    jy = torch.zeros_like(jx)
    for j in range(4):
        row = (iy - 1 + j) % ny * nx
        cum = torch.zeros_like(rx)
        for i in range(3):
            cum = cum + dx[i] * (sy[j] + 0.5 * dy[j])
            jx.index_add_(0, row + (ix - 1 + i) % nx, -p["q"] / dt * cum)
    for i in range(4):
        col = (ix - 1 + i) % nx
        cum = torch.zeros_like(rx)
        for j in range(3):
            cum = cum + dy[j] * (sx[i] + 0.5 * dx[i])
            jy.index_add_(0, (iy - 1 + j) % ny * nx + col, -p["q"] / dt * cum)
    return jx, jy


def _poisson64(rho, nx, ny, eig):
    spec = torch.fft.rfft2(rho.view(ny, nx))
    eig[0, 0] = 1.0
    spec = spec / eig
    spec[0, 0] = 0.0
    phi = torch.fft.irfft2(spec, s=(ny, nx))
    return phi, -(torch.roll(phi, -1, 1) - phi), -(torch.roll(phi, -1, 0) - phi)


def _modes(nx, ny):
    kw = dict(device=_device(), dtype=torch.float64)
    return 2.0 * math.pi * torch.fft.rfftfreq(nx, **kw)[None, :], 2.0 * math.pi * torch.fft.fftfreq(ny, **kw)[:, None]


def _step64(case, seed):
    nx, ny, dt, scheme = case["nx"], case["ny"], case["dt"], SCHEMES[case["scheme"]]
    p = _particles(case, seed)
    total, absolute = p["q"].sum(), p["q"].abs().sum()
    kx, ky = _modes(nx, ny)
    hist = []

    def push():
        p["x"] = torch.remainder(p["x"] + p["vx"] * dt, float(nx))
        p["y"] = torch.remainder(p["y"] + p["vy"] * dt, float(ny))

    for _ in range(case["steps"]):
        if scheme != ESK:
            push()
        rho = _deposit64(p, nx, ny, scheme, dt) + 1.0 / (nx * ny)
        phi, ex, ey = _poisson64(rho, nx, ny, kx * kx + ky * ky)
        if scheme == ESK:
            push()
        ix, rx = _split(p["x"], nx)
        iy, ry = _split(p["y"], ny)
        for v, e in (("vx", ex.reshape(-1)), ("vy", ey.reshape(-1))):
            at = 0.0
            for j, b in enumerate((1.0 - ry, ry)):
                for i, a in enumerate((1.0 - rx, rx)):
                    at = at + e[(iy + j) % ny * nx + (ix + i) % nx] * a * b
            p[v] = p[v] - p["q"] * at * dt
        ke = 0.5 * (p["vx"] ** 2 + p["vy"] ** 2).sum()
        fe = 0.5 * (ex ** 2 + ey ** 2).sum()
        err = (rho.sum() - total).abs() / absolute.clamp(min=1e-12)
        hist.append(torch.stack([err, total, rho.sum(), ke, fe, ke + fe]))
    fields = [rho, phi.reshape(-1), ex.reshape(-1), ey.reshape(-1)]
    return [torch.stack(hist)] + fields + ([None] * 5 if case["particles"] else [])


def _network64(case, seed):
    flat = _network_params(seed).double().to(_device())
    inp, tgt = (t.double()[:, None] for t in _network_fields(case, seed))
    at, params, shapes = 0, [], []
    for l, (ci, co) in enumerate(NET):
        cu, ou = (1 if l == 0 else ci), (1 if l == len(NET) - 1 else co)
        w = flat[at: at + 9 * co * ci].view(9, co, ci)
        b = flat[at + 9 * co * ci: at + 9 * co * ci + co]
        at += 9 * co * ci + co
        params.append((w[:, :ou, :cu].permute(1, 2, 0).reshape(ou, cu, 3, 3).clone().requires_grad_(),
                       b[:ou].clone().requires_grad_()))
        shapes.append((ci, co, cu, ou))
    loss, n = 0.0, inp.numel()
    for a, t in zip(inp, tgt):  # one sample at a time: the FP64 activations of all need not be kept
        h = a[None]
        for l, (w, b) in enumerate(params):
            h = torch.nn.functional.conv2d(torch.nn.functional.pad(h, (1, 1, 1, 1), mode="circular"), w, b)
            h = torch.relu(h) if l < len(params) - 1 else h
        part = ((h[0] - t) ** 2).sum() / n
        part.backward()
        loss += float(part)
    grad = []
    for (w, b), (ci, co, cu, ou) in zip(params, shapes):
        gw, gb = torch.zeros(9, co, ci, device=_device(), dtype=torch.float64), torch.zeros(co, device=_device(), dtype=torch.float64)
        gw[:, :ou, :cu] = w.grad.reshape(ou, cu, 9).permute(2, 0, 1)
        gb[:ou] = b.grad
        grad += [gw.reshape(-1), gb]
    return [loss, torch.cat(grad)]


def exact(case, seed):
    """What run() returns, in FP64. None for whole numbers and particle arrays (whose order
    follows the cell keys) and for the ensemble, whose particles the library itself draws."""
    kind = case["kind"]
    if kind in ("ensemble", "sort"):
        return None
    nx, ny = case["nx"], case["ny"]
    if kind == "call":
        return _deposit64(_particles(case, seed), nx, ny, SCHEMES[case["scheme"]], case["dt"])
    if kind == "deposit":
        return [_deposit64(_particles(case, seed), nx, ny, SCHEMES[case["scheme"]], case["dt"])]
    if kind == "esirkepov":
        p = _particles(case, seed)
        return [_deposit64(p, nx, ny, ESK, case["dt"]), *_current64(p, nx, ny, case["dt"])]
    if kind == "network":
        return _network64(case, seed)
    if kind == "rbgs":
        rho = _rbgs_rho(case, seed)
        kx, ky = _modes(nx, ny)
        fields = _poisson64(rho - rho.mean(), nx, ny, 4.0 - 2.0 * torch.cos(kx) - 2.0 * torch.cos(ky))
        return [None, None] + [f.reshape(-1) for f in fields]
    return _step64(case, seed)
