"""What a user has this library do, as cases that can be timed and compared.

Every case goes through the public entry points (the Solver class, and the C
ABI's device-pointer copies for state that lives on the GPU).  Three kinds:

  step      a coupled run of one or several domains: a cycle of a forecast or
            calibration loop that sets the head and the ponded depth from the
            program's own device arrays, prepares, advances, and reads the new
            state back into device arrays
  overland  the surface step alone, for a program that couples its own soil
            model: depth in, depth and elevation out
  adjoint   the calibration gradient: loss and dL/d(log Ks, alpha, n) per cell

Sizes are those of the benchmark workloads (32x32x20 FP64, 512x512x40 mixed,
the 16..128-wide uneven ensemble, 1024x1024x50, the 128x128x30 calibration
domain) and ragged ones between them.  Soil, surface and rain follow the same
distributions as dhara_b200.inputs; the state is one inside a storm: a water
table, a wetting front below the surface, pools in the hollows and a film of
water between them.  The 3D systems are solved to a residual of 1e-13, as the
calibration domain's gradient checks do.
"""
import ctypes as ct
import math
import random

import numpy as np
import torch

import dhara_b200 as db
from dhara_b200 import _abi

RAIN_MM_PER_H = 20.0
SOLVERS = dict(krylov_tol=1e-13, krylov_maxiter=1000, overland_tol=1e-12, overland_maxiter=4000)


def _step(name, nx, ny, nz, **kw):
    c = dict(name=name, kind="step", nx=nx, ny=ny, nz=nz, ndom=1, precision="mixed", steps=1, graph=False,
             soil="uniform", faces="closed", rule="absolute", theta="conservative", ks_sigma_ln=1.0)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest workload: launches, barriers and latency
        _step("step_32x32x20_fp64", 32, 32, 20, precision="fp64", ks_sigma_ln=0.5, steps=2, graph=True),
        # a drop-in caller's settings: the reference's Picard rule and moisture update, per-cell
        # soil, fixed heads on two sides, sizes that fit no tile
        _step("step_53x37x21_fp64_fixed", 53, 37, 21, precision="fp64", ks_sigma_ln=0.5, soil="cells",
              faces="fixed", rule="relative", theta="reference"),
        # the calibration domain's forward step
        _step("step_128x128x30", 128, 128, 30, ks_sigma_ln=0.5, graph=True),
        # a mid-size ragged catchment with per-cell soil
        _step("step_301x211x33_cells", 301, 211, 33, soil="cells"),
        # the headline domain, in both precisions
        _step("step_512x512x40", 512, 512, 40, graph=True),
        _step("step_512x512x40_fp64", 512, 512, 40, precision="fp64"),
        # the largest single domain
        _step("step_1024x1024x50", 1024, 1024, 50),
        # many uneven domains in one handle (16..128 columns a side, 20..40 layers)
        _step("ensemble_256", 128, 128, 40, ndom=256),
        # the surface alone: a plot and a catchment
        dict(name="overland_61x47", kind="overland", nx=61, ny=47),
        dict(name="overland_512x512", kind="overland", nx=512, ny=512),
        # the calibration gradient over two steps, one checkpoint segment each
        dict(name="adjoint_128x128x30", kind="adjoint", nx=128, ny=128, nz=30, steps=2, every=1),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "ensemble", "overland", "adjoint"])
    if kind == "overland":
        return dict(kind="overland", nx=log_int(40, 700), ny=log_int(40, 700))
    if kind == "adjoint":
        return dict(kind="adjoint", nx=log_int(24, 128), ny=log_int(24, 128), nz=rng.randint(12, 30),
                    steps=rng.randint(1, 2), every=rng.randint(1, 2))
    precision = rng.choice(["mixed", "mixed", "fp64"])
    side = 800 if precision == "mixed" else 550
    c = _step("", log_int(24, side), log_int(24, side), rng.randint(12, 50), precision=precision,
              graph=rng.random() < 0.5, soil=rng.choice(["uniform", "cells"]),
              ks_sigma_ln=round(rng.uniform(0.5, 1.0), 3), theta=rng.choice(["conservative", "conservative", "reference", "final"]))
    if kind == "ensemble":
        c.update(nx=log_int(32, 128), ny=log_int(32, 128), nz=rng.randint(21, 40), ndom=log_int(4, 200))
    elif c["nx"] * c["ny"] <= 200 * 200 and rng.random() < 0.4:
        c.update(faces="fixed")
    del c["name"]
    return c


# ------------------------------------------------------------------- inputs

def _sizes(case):
    """(nx, ny, nz) of every domain: the case's own, or uneven ones up to it."""
    nd = case.get("ndom", 1)
    nx, ny, nz = case["nx"], case["ny"], case.get("nz", 2)
    if nd == 1:
        return [(nx, ny, nz)]
    r = random.Random(nd * 1000003 + nx * 1009 + ny * 31 + nz)
    return [(r.randint(16, nx), r.randint(16, ny), r.randint(20, nz)) for _ in range(nd)]


def _params(case, nx, ny, nz):
    rule = dict(absolute=db.PICARD_PSI_ABSOLUTE, relative=db.PICARD_PSI_RELATIVE)[case.get("rule", "absolute")]
    theta = dict(conservative=db.THETA_CONSERVATIVE, reference=db.THETA_REFERENCE,
                 final=db.THETA_FINAL)[case.get("theta", "conservative")]
    adjoint = case["kind"] == "adjoint"
    kw = dict(alpha=3.5, n=1.6, theta_s=0.45, theta_r=0.05, porosity=0.45, Ss=5e-4, am=0.25,
              picard_rule=rule, picard_tol=1e-300 if adjoint else 1e-6, picard_maxiter=10, theta_update=theta,
              precision=db.FP64 if case.get("precision") == "fp64" else db.MIXED)
    kw.update(SOLVERS)
    return db.make_params(nx, ny, nz, dx=1.0, dy=1.0, dz=0.05, dt=60.0, **kw)


def _fields(p, case, seed):
    """One domain's seeded fields as FP64 device tensors in the reference layout."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    kw = dict(device="cuda", dtype=torch.float64)
    nx, ny, nz = p.nx, p.ny, p.nz
    # micro-topography: a Gaussian random field, sigma 5 cm, correlation 3 m, on a 1 % slope
    mx, my = nx + 9, ny + 9
    kx = 2 * math.pi * torch.fft.fftfreq(mx, d=p.dx, **kw)
    ky = 2 * math.pi * torch.fft.fftfreq(my, d=p.dy, **kw)
    spec = torch.exp(-(ky[:, None] ** 2 + kx[None, :] ** 2) * 9.0 / 8.0)
    f = torch.fft.ifft2(torch.fft.fft2(torch.randn(my, mx, generator=g, **kw)) * spec).real[:ny, :nx]
    f = f - f.mean()
    f = f * (0.05 / f.std())
    z = 1.0 + 0.01 * p.dx * torch.arange(nx - 1, -1, -1, **kw)[None, :] + f
    # pools in the hollows, a thin uneven film elsewhere
    film = 5e-4 * torch.rand(ny, nx, generator=g, **kw)
    ponding = torch.clamp(-0.6 * (f + 0.03), min=0.0) + film
    out = dict(ztopo=z, mann=torch.full((ny, nx), 0.03, **kw), ponding=ponding)
    if case["kind"] == "overland":
        return out
    out["ksat"] = 1e-5 * torch.exp(case.get("ks_sigma_ln", 0.5) * torch.randn(nz, ny, nx, generator=g, **kw))
    # hydrostatic over a water table at 0.8 m, a wetting front of uneven strength below the surface
    depth = (torch.arange(nz, **kw) + 0.5) * p.dz
    front = 0.3 + 0.3 * torch.rand(ny, nx, generator=g, **kw)
    out["psi"] = (depth - 0.8)[:, None, None] + front[None] * torch.exp(-depth / 0.15)[:, None, None]
    if case.get("soil") == "cells":
        out["alpha"] = 3.5 * torch.exp(0.1 * torch.randn(nz, ny, nx, generator=g, **kw))
        out["nvg"] = 1.6 + 0.1 * (torch.rand(nz, ny, nx, generator=g, **kw) - 0.5)
    return {k: v.contiguous() for k, v in out.items()}


def _rain(p, steps):
    return np.full(steps, RAIN_MM_PER_H * p.dt / 3600.0)


def _fixed_faces(solver, p, psi, domain=0):
    """Fixed heads on the west and south faces: the initial profile's."""
    west = psi[:, :, 0].cpu().numpy().reshape(-1)
    south = psi[:, 0, :].cpu().numpy().reshape(-1)
    solver.upload("bcw", np.zeros(west.size, np.int32), domain)
    solver.upload("bcs", np.zeros(south.size, np.int32), domain)
    solver.upload("bcpsiw", west, domain)
    solver.upload("bcpsis", south, domain)


def _put(solver, name, t, domain=0):
    rc = db.lib().dhara_upload_device(solver.h, domain, _abi.F[name], ct.c_void_p(t.data_ptr()), ct.c_int64(t.numel()))
    if rc:
        raise db.DharaError(rc, db.lib().dhara_last_error().decode())


def _get(solver, name, t, domain=0):
    rc = db.lib().dhara_download_device(solver.h, domain, _abi.F[name], ct.c_void_p(t.data_ptr()),
                                        ct.c_int64(t.numel()))
    if rc:
        raise db.DharaError(rc, db.lib().dhara_last_error().decode())
    return t


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    sizes = _sizes(case)
    plist = [_params(case, *n) for n in sizes]
    fields = [_fields(p, case, seed * 4099 + d) for d, p in enumerate(plist)]
    torch.cuda.synchronize()  # the solver works on a stream of its own
    s.solver = db.Solver(plist)
    s.set_each, s.out = [], []
    like = torch.empty_like
    for d, (p, f) in enumerate(zip(plist, fields)):
        if case["kind"] == "overland":
            f["psi"] = torch.full((p.nz, p.ny, p.nx), -0.5, device="cuda", dtype=torch.float64)
            f["ksat"] = torch.full_like(f["psi"], 1e-5)
        for k in ("ztopo", "mann", "ksat", "psi", "ponding"):
            _put(s.solver, k, f[k], d)
        if case.get("soil") == "cells":
            for k in ("alpha", "nvg"):
                s.solver.upload(k, f[k].cpu().numpy().reshape(-1), d)
        if case["kind"] != "overland":
            s.solver.set_rain_schedule(_rain(p, case["steps"]), d)
        if case.get("faces") == "fixed":
            _fixed_faces(s.solver, p, f["psi"], d)
        if case["kind"] == "overland":
            s.set_each.append({"waterdepth": f["ponding"]})
            s.out.append({"waterdepth": like(f["ponding"]), "waterelev": like(f["ponding"])})
        else:
            s.set_each.append({"psi": f["psi"], "ponding": f["ponding"]})
            if case["kind"] == "step":
                s.out.append({"psi": like(f["psi"]), "theta": like(f["psi"]), "waterdepth": like(f["ponding"]),
                              "waterelev": like(f["ponding"])})
    if case["kind"] == "adjoint":
        # observed moisture of the top three layers and outflow, as a calibration run has them
        p, n = plist[0], case["steps"]
        g = np.random.default_rng(seed)
        s.theta_target = 0.25 + 0.1 * g.random((n, 3 * p.nx * p.ny))
        s.q_target = 1e-3 * g.random(n)
    if case["kind"] == "step" and case["ndom"] > 16:
        # a many-domain program gathers its results in one array per quantity
        s.whole = {}
        for k in s.out[0]:
            s.whole[k] = torch.empty(sum(o[k].numel() for o in s.out), device="cuda", dtype=torch.float64)
            at = 0
            for o in s.out:
                o[k] = s.whole[k][at:at + o[k].numel()]
                at += o[k].numel()
    s.solver.prepare()
    return s


def run(s):
    for d, fields in enumerate(s.set_each):
        for k, t in fields.items():
            _put(s.solver, k, t, d)
    kind = s.case["kind"]
    if kind == "overland":
        s.solver.overland_step()
        return {k: _get(s.solver, k, t) for k, t in s.out[0].items()}
    s.solver.prepare()
    if kind == "adjoint":
        loss, g_ks, g_alpha, g_n = s.solver.adjoint(s.theta_target, s.q_target, s.case["steps"], s.case["every"],
                                                    w_q=1.0)
        return {"loss": loss, "log_ks": g_ks, "alpha": g_alpha, "n": g_n}
    s.solver.step(s.case["steps"], s.case["graph"])
    for d, o in enumerate(s.out):
        for k, t in o.items():
            _get(s.solver, k, t, d)
    if s.case["ndom"] > 16:
        return s.whole
    return s.out[0] if len(s.out) == 1 else s.out


def work(case):
    """The least a pass has to move and compute.  A step: per Picard iteration
    (at the cap of 10, which these states reach or nearly reach) psi^m, psi^n,
    theta^n and Ks read and the new head written, and one linear solve that
    reads its matrix (storage diagonal, conductivity) and right-hand side once
    per iteration of a Krylov method, a dozen iterations at least for twelve
    digits.  The surface: about forty iterations over its five-point rows."""
    surface = sum(nx * ny for nx, ny, _ in _sizes(case))
    if case["kind"] == "overland":
        return {"bytes": 8.0 * 5 * surface, "flops": 40.0 * 40 * surface}
    cells = sum(nx * ny * nz for nx, ny, nz in _sizes(case))
    word = 8 if case.get("precision") == "fp64" else 4
    per_solve = 5 * 8 + 12 * 3 * word
    solves = 10.0 * case["steps"] * (3 if case["kind"] == "adjoint" else 1)
    return {"bytes": cells * per_solve * solves + 8.0 * 5 * surface * case["steps"],
            "flops": cells * (12 * 40 + 150) * solves + 40.0 * 40 * surface * case["steps"]}


# --------------------------------------------------------- 64-bit reference

def exact(case, seed):
    """The same step in plain torch FP64: the reference's modified Picard
    iteration (src/subsurface.cu:686-847) and overland step
    (src/overland.cu:387-419) with every linear system solved to rounding.
    Closed side faces and single domains (fixed faces, ensembles and gradients
    have no such value here)."""
    if case["kind"] == "adjoint" or case.get("ndom", 1) > 1 or case.get("faces") == "fixed":
        return None
    nx, ny, nz = _sizes(case)[0]
    p = _params(case, nx, ny, nz)
    f = _fields(p, case, seed * 4099)
    if case["kind"] == "overland":
        depth, elev = _exact_overland(p, f["ponding"], f["ztopo"], f["mann"])
        return {"waterdepth": depth, "waterelev": elev}
    psi, ponding = f["psi"], f["ponding"]
    alpha, n = f.get("alpha", p.alpha), f.get("nvg", p.n)
    ks = f["ksat"]

    def closure(h):
        x = alpha * torch.clamp(-h, min=1e-300)
        m = 1.0 - 1.0 / n
        xn = x ** n
        se = torch.exp(-m * torch.log1p(xn))
        lq = torch.where(xn > 1.0, -torch.log1p(1.0 / xn), n * torch.log(x) - torch.log1p(xn))
        kr = -torch.expm1(m * lq)
        wet = h >= 0
        th = torch.where(wet, p.theta_s, p.theta_r + (p.theta_s - p.theta_r) * se)
        k = torch.where(wet, ks, ks * torch.sqrt(se) * kr * kr)
        c = torch.where(wet, 0.0, alpha * (n - 1.0) * (p.theta_s - p.theta_r) * x ** (n - 1.0) * se / (1.0 + xn))
        return th, k, c

    dt, dz = p.dt, p.dz
    ssc = p.Ss / dt / p.porosity
    theta, k, _ = closure(psi)
    ktop, x = k[0].clone(), psi.clone()
    for rain in _rain(p, case["steps"]):
        hpot = ponding + rain / 1000.0
        qcapa = -ktop * ((psi[0] - hpot - 0.5 * dz) / (0.5 * dz))
        qcapa = torch.where(ponding / dt > ks[0], torch.maximum(qcapa, ks[0]), qcapa)
        q = torch.minimum(torch.minimum(torch.minimum(hpot / dt, qcapa), (p.theta_s - theta[0]) * dz / dt), ks[0])
        q = torch.where(hpot > 0, q, hpot / dt)
        x = psi.clone()
        for it in range(p.picard_maxiter):
            pm = psi if it == 0 else p.am * pm + (1.0 - p.am) * x
            th, k, c = closure(pm)
            fz = 0.5 * (k[1:] + k[:-1])
            rhs = ssc * th * psi + c / dt * pm + (theta - th) / dt
            rhs[:-1] -= fz / dz
            rhs[1:] += fz / dz
            rhs[0] += q / dz
            rhs[-1] -= k[-1] / dz
            x = _solve3d(p, ssc * th + c / dt, k, rhs, x)
            d = (x - pm).abs()
            if p.picard_rule == db.PICARD_PSI_RELATIVE:
                d = d / x.abs()
            if d.max() < p.picard_tol:
                break
        th1, k1, _ = closure(x)
        if p.theta_update == db.THETA_FINAL:
            theta = th1
        elif p.theta_update == db.THETA_CONSERVATIVE:
            theta = th + c * (x - pm)
        else:
            theta = th
        psi, ktop = x, k1[0].clone()
        ponding, elev = _exact_overland(p, torch.clamp(hpot - q * dt, min=0.0), f["ztopo"], f["mann"])
    return {"psi": psi, "theta": theta, "waterdepth": ponding, "waterelev": elev}


def _solve3d(p, diag, k, rhs, x):
    """Conjugate gradients preconditioned by every column's tridiagonal block,
    restarted from the true residual until that stops falling."""
    fx = 0.5 * (k[:, :, 1:] + k[:, :, :-1]) / p.dx ** 2
    fy = 0.5 * (k[:, 1:] + k[:, :-1]) / p.dy ** 2
    fz = 0.5 * (k[1:] + k[:-1]) / p.dz ** 2
    nz = k.shape[0]

    def apply(v):
        out = diag * v
        d = fx * (v[:, :, 1:] - v[:, :, :-1])
        out[:, :, :-1] -= d
        out[:, :, 1:] += d
        d = fy * (v[:, 1:] - v[:, :-1])
        out[:, :-1] -= d
        out[:, 1:] += d
        d = fz * (v[1:] - v[:-1])
        out[:-1] -= d
        out[1:] += d
        return out

    b = diag.clone()
    for face, cut in ((fx, lambda t, s: t[:, :, s]), (fy, lambda t, s: t[:, s]), (fz, lambda t, s: t[s])):
        cut(b, slice(None, -1)).add_(face)
        cut(b, slice(1, None)).add_(face)
    inv, cp = torch.empty_like(b), torch.zeros_like(b)
    for i in range(nz):
        den = b[i] if i == 0 else b[i] + fz[i - 1] * cp[i - 1]
        inv[i] = 1.0 / den
        if i + 1 < nz:
            cp[i] = -fz[i] * inv[i]

    def column(r):
        y = r.clone()
        for i in range(1, nz):
            y[i] -= cp[i - 1] * y[i - 1]
        y *= inv
        for i in range(nz - 2, -1, -1):
            y[i] -= cp[i] * y[i + 1]
        return y

    last = math.inf
    for _ in range(4):
        r = rhs - apply(x)
        now = float(r.norm() / rhs.norm())
        if now < 1e-15 or now > 0.5 * last:
            break
        last = now
        d = torch.zeros_like(x)
        z = column(r)
        v, rz = z.clone(), (r * z).sum()
        stop = float(rz) * 1e-18
        for it in range(400):
            q = apply(v)
            a = rz / (v * q).sum()
            d += a * v
            r -= a * q
            z = column(r)
            new = (r * z).sum()
            if it % 4 == 3 and float(new) <= stop:
                break
            v = z + (new / rz) * v
            rz = new
        x = x + d
    return x


def _exact_overland(p, depth, z, mann):
    """Manning conductances and the implicit five-point system on the interior,
    the outer ring fixed, by diagonally scaled conjugate gradients."""
    h = depth + z
    kx = torch.zeros(p.ny, p.nx - 1, device=z.device, dtype=z.dtype)  # the face between (j, i) and (j, i + 1)
    ky = torch.zeros(p.ny - 1, p.nx, device=z.device, dtype=z.dtype)

    def conductance(a, b, along, across, ha, hb, ma, mb):
        s = torch.sqrt(along ** 2 + across ** 2)
        up = torch.where(hb > ha, b, a)
        mid = 0.5 * (a + b)
        flows = (up > p.hmin) & (mid > p.hmin) & (s > p.delta)
        k = torch.clamp(mid, min=0.0) ** (5.0 / 3.0) / (0.5 * (ma + mb) * torch.sqrt(torch.clamp(s, min=1e-300)))
        return torch.where(flows, k, p.K0)

    across = (h[2:, 1:] + h[2:, :-1] - h[:-2, 1:] - h[:-2, :-1]) / (4 * p.dy)
    m = slice(1, -1)
    kx[m] = conductance(depth[m, :-1], depth[m, 1:], (h[m, 1:] - h[m, :-1]) / p.dx, across, h[m, :-1], h[m, 1:],
                        mann[m, :-1], mann[m, 1:])
    across = (h[1:, 2:] + h[:-1, 2:] - h[1:, :-2] - h[:-1, :-2]) / (4 * p.dx)
    ky[:, m] = conductance(depth[:-1, m], depth[1:, m], (h[1:, m] - h[:-1, m]) / p.dy, across, h[:-1, m], h[1:, m],
                           mann[:-1, m], mann[1:, m])
    cx, cy = p.dt / p.dx ** 2 * kx, p.dt / p.dy ** 2 * ky

    def apply(v):  # interior rows
        c = v[1:-1, 1:-1]
        return c + (cx[1:-1, 1:] * (c - v[1:-1, 2:]) + cx[1:-1, :-1] * (c - v[1:-1, :-2])
                    + cy[1:, 1:-1] * (c - v[2:, 1:-1]) + cy[:-1, 1:-1] * (c - v[:-2, 1:-1]))

    if p.nx > 2 and p.ny > 2:
        dg = 1.0 + cx[1:-1, 1:] + cx[1:-1, :-1] + cy[1:, 1:-1] + cy[:-1, 1:-1]
        b = h[1:-1, 1:-1].clone()
        x = h.clone()
        last = math.inf
        for _ in range(4):
            r = b - apply(x)
            now = float(r.norm() / b.norm())
            if now < 1e-15 or now > 0.5 * last:
                break
            last = now
            v = torch.zeros_like(x)
            e = torch.zeros_like(b)
            u = r / dg
            v[1:-1, 1:-1] = u
            g = (r * u).sum()
            stop = float(g) * 1e-20
            for it in range(8000):
                q = apply(v)
                a = g / (v[1:-1, 1:-1] * q).sum()
                e += a * v[1:-1, 1:-1]
                r -= a * q
                u = r / dg
                new = (r * u).sum()
                if it % 16 == 15 and float(new) <= stop:
                    break
                v[1:-1, 1:-1] = u + (new / g) * v[1:-1, 1:-1]
                g = new
            x[1:-1, 1:-1] += e
        h = x
    return torch.clamp(h - z, min=0.0), h
