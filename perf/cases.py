"""The workloads whose speed this framework is judged by, through its public entry points.

Each case is one call (or one short run) of the host API in pmf-glm_b200/pmfmhd.py on a
periodic turbulent box of the benchmark's kind: density 1 + 0.1 g, velocity rms Mach 0.5, a
magnetic field of plasma beta 1, all Gaussian random fields (cut at an eighth of the grid's
modes, so that the turbulence is resolved). ``listed`` names the workloads,
``draw`` gives more of the same ranges, ``prepare`` makes a state on the GPU from a seed,
``run`` takes one pass, ``work`` counts what a pass cannot do without, and ``exact`` restates
the scheme in 64-bit torch for the error of the result.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pmf-glm_b200"))

import pmfmhd  # noqa: E402

GAMMA, CFL, CR = 5.0 / 3.0, 0.2, 0.18
SMALLR, PFL, DTOL = 1e-6, 1e-7, 1e-5
DEV = "cuda"


def _box(kind, nx, ny=None, nz=None, **kw):
    c = dict(kind=kind, nx=nx, ny=ny or nx, nz=nz or nx, recon="plm", riemann="hlld", bx="periodic", by="periodic",
             bz="periodic", solver="glm", compensated=False)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest box of the batched configuration, stepped alone: latency and launches
        dict(name="glm_32", **_box("step", 32)),
        # the 64^3 plain configuration driven the way a run drives it: evolve() picks dt each step
        dict(name="evolve_64", **_box("evolve", 64)),
        # a ragged box with walls and the PPM / HLL options of the reference's tests
        dict(name="glm_ppm_hll_ragged", **_box("step", 100, 75, 61, recon="ppm", riemann="hll", bx="outflow",
                                               by="reflecting")),
        # the headline box
        dict(name="glm_256", **_box("step", 256)),
        # the precision form: compensated update on the largest configuration
        dict(name="glm_comp_512", **_box("step", 512, compensated=True)),
        # constrained transport, a small box of the batched configuration stepped alone
        dict(name="ct_48", **_box("step", 48, solver="ct")),
        # constrained transport on the headline box
        dict(name="ct_256", **_box("step", 256, solver="ct")),
        # the drag-coupled step of the production runner on a box that is no multiple of a tile
        dict(name="drag_ragged", **_box("drag", 150, 131, 96)),
        # the radiation-coupled step of the production runner with its tracking on
        dict(name="rad_128", **_box("rad", 128)),
        # the batched form: uneven GLM and CT boxes, dt on the device
        dict(name="batch_64", kind="batch", boxes=64, largest=128, seed_mix=2024),
        # terminal-regime induction of a CT state, one SSPRK2 subcycle, order-4 dissipation
        dict(name="terminal_ct_128", **_box("terminal", 128, solver="ct", order=4)),
        # the ledger and the div-B norm of the headline box
        dict(name="ledger_256", **_box("ledger", 256)),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "ct", "ct", "drag", "rad", "evolve", "batch", "terminal", "ledger"])
    if kind == "batch":
        return dict(kind="batch", boxes=size(8, 64), largest=rng.choice([64, 96, 128]), seed_mix=rng.randrange(1 << 30))
    if kind in ("terminal",):
        return _box("terminal", size(24, 160), solver=rng.choice(["glm", "ct"]), order=rng.choice([2, 4]))
    if kind == "evolve":
        n = size(24, 128)
        return _box("evolve", n, solver=rng.choice(["glm", "glm", "ct"]))
    dims = [size(24, 224)] * 3 if rng.random() < 0.5 else [size(20, 224) for _ in range(3)]
    recon = rng.choice(["plm", "plm", "plm", "ppm", "plm_minmod"])
    riemann = rng.choice(["hlld", "hlld", "hlld", "hll", "llf"])
    if kind == "ct":
        return _box("step", *dims, solver="ct", recon=recon, riemann=riemann)
    if kind == "step":
        walls = [rng.choice(["periodic", "periodic", "outflow", "reflecting"]) for _ in range(3)]
        return _box("step", *dims, recon=recon, riemann=riemann, bx=walls[0], by=walls[1], bz=walls[2],
                    compensated=rng.random() < 0.3)
    return _box(kind, *dims)


# ---- inputs ------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _grf(shape, gen, index, kcut):
    """Gaussian random field of unit variance, P(k) ~ k^index up to mode number kcut (in modes
    of the longest side)."""
    w = torch.fft.rfftn(torch.randn(shape, generator=gen, device=DEV))
    n = max(shape)
    k2 = 0
    for ax, m in enumerate(shape):
        f = torch.fft.rfftfreq(m, device=DEV) if ax == 2 else torch.fft.fftfreq(m, device=DEV)
        k2 = k2 + (f * n).square().reshape([-1 if a == ax else 1 for a in range(3)])
    amp = torch.where((k2 > 0) & (k2 <= kcut * kcut), k2.clamp(min=1e-12).pow(index / 4), torch.zeros_like(k2))
    f = torch.fft.irfftn(w.mul_(amp), s=shape)
    f -= f.mean()
    return f / f.square().mean().sqrt()


def _up(a, ax):
    return torch.roll(a, -1, ax)


def _dn(a, ax):
    return torch.roll(a, 1, ax)


def _fields(shape, seed, solver, beta=1.0, index=2.0, kc=None):
    """The conserved fields (nine float32 arrays) and, for CT, the three lower-face fields."""
    gen = _gen(seed)
    n = max(shape)
    rho = 1.0 + 0.1 * _grf(shape, gen, -2.0, n / 8).clamp(-5, 5)
    # a bulk drift; of a CT box large enough that the mass flux whose sign picks the upwind side of
    # an edge EMF vanishes almost nowhere (a zero crossing there is a jump that rounding decides)
    drift = (1.0, -0.9, 0.95) if solver == "ct" else (0.1, -0.05, 0.08)
    v = [_grf(shape, gen, -2.0, n / 8) * (0.5 / math.sqrt(3)) + d for d in drift]
    A = [_grf(shape, gen, index - 2.0, kc or min(16.0, n / 8)) for _ in range(3)]
    faces = None
    if solver == "ct":  # staggered curl of an edge potential, cell B its face average
        faces = [(_up(A[2], 1) - A[2]) - (_up(A[1], 0) - A[1]), (_up(A[0], 0) - A[0]) - (_up(A[2], 2) - A[2]),
                 (_up(A[1], 2) - A[1]) - (_up(A[0], 1) - A[0])]
        B = [0.5 * (f + _up(f, 2 - d)) for d, f in enumerate(faces)]
    else:
        dc = lambda a, ax: _up(a, ax) - _dn(a, ax)  # noqa: E731
        B = [dc(A[2], 1) - dc(A[1], 0), dc(A[0], 0) - dc(A[2], 2), dc(A[1], 2) - dc(A[0], 1)]
    p0 = 1.0 / GAMMA
    s = (2.0 * p0 / beta / sum(b.square().mean() for b in B)).sqrt()
    if faces is not None:
        faces = [f * s for f in faces]
        B = [0.5 * (f + _up(f, 2 - d)) for d, f in enumerate(faces)]
    else:
        B = [b * s for b in B]
    E = p0 / (GAMMA - 1) + 0.5 * rho * sum(c.square() for c in v) + 0.5 * sum(b.square() for b in B)
    return [rho, rho * v[0], rho * v[1], rho * v[2], E, *B, torch.zeros_like(rho)], faces


def _terminal_fields(shape, seed, solver):
    """Overdamped gas: density near 1, a field of rms 0.08 and thermal energy 1.5, at rest."""
    U, faces = _fields(shape, seed, solver)
    s = 0.08 / math.sqrt(2 / GAMMA)
    if faces is not None:
        faces = [f * s for f in faces]
        B = [0.5 * (f + _up(f, 2 - d)) for d, f in enumerate(faces)]
    else:
        B = [b * s for b in U[5:8]]
    z = torch.zeros_like(U[0])
    return [0.8 + 0.2 * U[0], z, z, z, 1.5 + 0.5 * sum(b.square() for b in B), *B, z], faces


def _f32(x):
    return float(np.float32(x))


def _shape(c):
    return (c["nz"], c["ny"], c["nx"])


def _dx(c):
    return _f32(1.0 / max(c["nx"], c["ny"], c["nz"]))


def _inputs(c, seed):
    """Fields, faces and the scalars of the call, by torch alone."""
    if c["kind"] == "terminal":
        U, faces = _terminal_fields(_shape(c), seed, c["solver"])
        vmax = float(sum(v.square() for v in _terminal_velocity([u.double() for u in U], U[5:8], _dx(c))).max().sqrt())
        return U, faces, dict(dt=_f32(0.9 * 0.4 * _dx(c) / vmax))  # one subcycle
    U, faces = _fields(_shape(c), seed, c["solver"])
    smax = 0.0
    for k in range(0, c["nz"], 32):
        smax = max(smax, _wavespeed([u[k:k + 32].double() for u in U]))
    ch, dt = _f32(smax), _f32(CFL * _dx(c) / smax)
    return U, faces, dict(dt=dt, ch=ch, decay=_f32(math.exp(-CR * ch * dt / _dx(c))))


def _mix(c):
    """Side lengths, solvers and field parameters of the batched workload."""
    rng = np.random.default_rng(c["seed_mix"])
    sizes = [n for n in (32, 48, 64, 96, 128) if n <= c["largest"]]
    p = np.array((5, 4, 3, 2, 1)[:len(sizes)], dtype=float)
    out = []
    for i in range(c["boxes"]):
        n = c["largest"] if i == 0 else int(rng.choice(sizes, p=p / p.sum()))
        out.append(dict(n=n, beta=float(10 ** rng.uniform(-1.0, 1.0)), index=float(rng.uniform(-2.9, 2.0)),
                        kc=float(rng.uniform(n / 16, n / 8)), solver="ct" if rng.integers(0, 2) else "glm"))
    return out


def _load(s, U, faces):
    for a, u in zip(s.U, U):
        a.copy_(u.reshape(-1))
    if faces is not None:
        s.ct.packed[:3 * s.nc].copy_(torch.stack([f.reshape(-1) for f in faces]).reshape(-1))
    return s


def prepare(case, seed):
    if case["kind"] == "batch":
        boxes, specs = [], _mix(case)
        flat = torch.zeros(9 * sum(b["n"] ** 3 for b in specs), device=DEV)  # all boxes' fields
        packed = torch.zeros(21 * sum(b["n"] ** 3 for b in specs if b["solver"] == "ct"), device=DEV)
        a = q = 0
        for i, b in enumerate(specs):
            n, nc = b["n"], b["n"] ** 3
            s = pmfmhd.allocate_state((n, n, n), 1.0 / n, mhd_solver=b["solver"])
            s.U = [flat[a + v * nc:a + (v + 1) * nc] for v in range(9)]
            a += 9 * nc
            if b["solver"] == "ct":
                s.ct = pmfmhd.CTState(packed[q:q + 21 * nc], nc)
                q += 21 * nc
            boxes.append(_load(s, *_fields((n, n, n), seed * 1000 + i, b["solver"], b["beta"], b["index"], b["kc"])))
        return dict(kind="batch", batch=pmfmhd.Batch(boxes, cfl=CFL), flat=flat,
                    faces=[s.ct.packed[:3 * s.nc] for s in boxes if s.ct is not None])
    U, faces, par = _inputs(case, seed)
    s = pmfmhd.allocate_state((case["nx"], case["ny"], case["nz"]), _dx(case), recon=case["recon"],
                              riemann=case["riemann"], bcs=(case["bx"], case["by"], case["bz"]),
                              mhd_solver=case["solver"], compensated=case["compensated"])
    st = dict(kind=case["kind"], s=_load(s, U, faces), order=case.get("order"), **par)
    if case["kind"] == "evolve":
        st["tfinal"] = 3.5 * par["dt"]  # four steps
    if case["kind"] == "rad":
        st["corr"] = pmfmhd.allocate_radiation_correction(s)
        for d, v in enumerate(_corrections(case, seed)):
            st["corr"][(1 + d) * s.nc:(2 + d) * s.nc].copy_(v.reshape(-1))
    return st


def _corrections(c, seed):
    gen = _gen(seed + 77)
    return [2e-3 * _grf(_shape(c), gen, -2.0, max(_shape(c)) / 8) for _ in range(3)]


def run(st):
    k = st["kind"]
    if k == "batch":
        st["batch"].step(2)  # two steps: the current state is back in the boxes' first buffers
        return [st["flat"], torch.cat(st["faces"]) if st["faces"] else st["flat"][:0]]
    s = st["s"]
    ct = s.ct is not None
    if k == "step":
        pmfmhd.step(s, st["dt"], ch=st["ch"], integrator="ref" if ct else "cube")
    elif k == "evolve":
        _, n = pmfmhd.evolve(s, st["tfinal"], cfl=CFL)
    elif k == "drag":
        pmfmhd.step_drag_godunov(s, st["dt"], 0.05, st["ch"])
    elif k == "rad":
        # the runner refreshes psi in the correction buffer before each step
        st["corr"][:s.nc].copy_(s.U[8])
        pmfmhd.step_cube_radiation(s, st["dt"], st["ch"], st["decay"], 0.05, st["corr"], check_admissibility=True)
        return [*s.U, st["corr"][4 * s.nc:5 * s.nc]]
    elif k == "terminal":
        pmfmhd.terminal_ct_induction(s, st["dt"], 4.0, 0.2, dissipation_order=st["order"])
        return [s.U[0], s.U[4], s.U[5], s.U[6], s.U[7]] + ([s.ct.packed[:3 * s.nc]] if ct else [])
    elif k == "ledger":
        t = pmfmhd.conserved_totals(s)
        return [np.array(list(t.values())), np.float64(pmfmhd.max_divb(s))]
    # (the Kahan remainders of a compensated state are the part of its value below one rounding
    # unit: they hold nothing that a second rounding would reproduce)
    return [*s.U] + ([s.ct.packed[:3 * s.nc]] if ct else []) + ([n] if k == "evolve" else [])


def work(case):
    """Compulsory bytes and operations. Per zone of a step: about 160 for the limited slopes, 250
    for the predictor, 230 for each of three HLLD faces, 100 for the update and signal speed."""
    glm, ct = 72, 72 - 12 + 24  # fields in and out; CT: no cell B written by the stage, faces in and out
    k = case["kind"]
    if k == "batch":
        per = [(b["n"] ** 3, ct + 12 if b["solver"] == "ct" else glm) for b in _mix(case)]
        return {"bytes": 2 * sum(n * b for n, b in per), "flops": 2 * 1200 * sum(n for n, _ in per)}
    nc = case["nx"] * case["ny"] * case["nz"]
    step = ct + 12 if case["solver"] == "ct" else glm
    if k == "evolve":
        return {"bytes": 4 * step * nc, "flops": 4 * 1200 * nc}
    if k == "terminal":  # rho, E, B (and faces) in; E, B (and faces and remainders) out
        return {"bytes": (36 + (48 if case["solver"] == "ct" else 0)) * nc, "flops": 400 * nc}
    if k == "ledger":
        return {"bytes": 32 * nc, "flops": 20 * nc}
    extra = 56 if case["compensated"] else 12 + 8 + 24 + 8 if k == "rad" else 0
    return {"bytes": (step + extra) * nc, "flops": 1200 * nc}


# ---- the same in 64-bit torch ------------------------------------------------------------

def _prim(U):
    rho = U[0].clamp(min=SMALLR)
    v = [U[c] / rho for c in (1, 2, 3)]
    p = (GAMMA - 1) * (U[4] - 0.5 * (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / rho - 0.5 * (U[5] ** 2 + U[6] ** 2 + U[7] ** 2))
    return [rho, *v, p.clamp(min=PFL), U[5], U[6], U[7], U[8]]


def _cons(q):
    E = q[4] / (GAMMA - 1) + 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2) + 0.5 * (q[5] ** 2 + q[6] ** 2 + q[7] ** 2)
    return [q[0], q[0] * q[1], q[0] * q[2], q[0] * q[3], E, q[5], q[6], q[7], q[8]]


def _fast(q, bn):
    c2 = GAMMA * q[4] / q[0]
    d2 = 0.5 * ((q[5] ** 2 + q[6] ** 2 + q[7] ** 2) / q[0] + c2)
    return (d2 + (d2 * d2 - c2 * bn * bn / q[0]).clamp(min=0).sqrt()).sqrt()


def _wavespeed(U):
    q = _prim(U)
    return max(float((q[1 + d].abs() + _fast(q, q[5 + d])).max()) for d in range(3))


_PERM = ((0, 1, 2, 3, 4, 5, 6, 7, 8), (0, 2, 3, 1, 4, 6, 7, 5, 8), (0, 3, 1, 2, 4, 7, 5, 6, 8))


def _rot(q, D):
    return [q[j] for j in _PERM[D]]


def _back(f, D):
    out = [None] * 9
    for i, j in enumerate(_PERM[D]):
        out[j] = f[i]
    return out


def _flux(q):
    rho, u, v, w, p, bx, by, bz, _ = q
    b2 = bx * bx + by * by + bz * bz
    pt = p + 0.5 * b2
    E = p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v + w * w) + 0.5 * b2
    z = torch.zeros_like(rho)
    return [rho * u, rho * u * u + pt - bx * bx, rho * u * v - bx * by, rho * u * w - bx * bz,
            (E + pt) * u - bx * (u * bx + v * by + w * bz), z, u * by - v * bx, u * bz - w * bx, z]


def _offsets(m, c, p, recon):
    if recon == "ppm":
        slope, curve = (p - m) * 0.25, (m - 2 * c + p) / 12
        qL, qR = c - slope + curve, c + slope + curve
        dq, mid = qR - qL, 0.5 * (qL + qR)
        diff = (c - mid) * dq
        flat, over, under = (qR - c) * (c - qL) <= 0, diff > dq * dq / 6, diff < -dq * dq / 6
        L = torch.where(over, 3 * c - 2 * qR, qL)
        R = torch.where(~over & under, 3 * c - 2 * qL, qR)
        return torch.where(flat, c, L) - c, torch.where(flat, c, R) - c
    dl, dr = c - m, p - c
    lim = torch.minimum(dl.abs(), dr.abs())
    if recon == "plm":
        lim = torch.minimum(2 * lim, 0.5 * (dl + dr).abs())
    h = 0.5 * torch.where(dl * dr > 0, torch.sign(dl) * lim, torch.zeros_like(lim))
    return -h, h


def _riemann(L, R, D, ch, riemann, bn=None):
    """Flux through a D-normal face; bn: the staggered field (constrained transport)."""
    L, R = _rot(L, D), _rot(R, D)
    for q in (L, R):
        q[0], q[4] = q[0].clamp(min=SMALLR), q[4].clamp(min=PFL)
    if bn is None:
        bs = 0.5 * (L[5] + R[5]) - 0.5 * (R[8] - L[8]) / ch
        ps = 0.5 * (L[8] + R[8]) - 0.5 * ch * (R[5] - L[5])
        fb, fp = ps, ch * ch * bs
    else:
        bs, fb, fp = bn, torch.zeros_like(bn), torch.zeros_like(bn)
    L[5] = R[5] = bs
    fL, fR = _flux(L), _flux(R)
    uL, uR = _cons(L), _cons(R)
    cL, cR = _fast(L, bs), _fast(R, bs)
    if riemann == "llf":
        s = torch.maximum(L[1].abs() + cL, R[1].abs() + cR).clamp(min=ch)
        f = [0.5 * (a + b) - 0.5 * s * (d - c) for a, b, c, d in zip(fL, fR, uL, uR)]
    elif riemann == "hll":
        SL, SR = torch.minimum(L[1] - cL, R[1] - cR).clamp(max=0), torch.maximum(L[1] + cL, R[1] + cR).clamp(min=0)
        f = [(SR * a - SL * b + SL * SR * (d - c)) / (SR - SL) for a, b, c, d in zip(fL, fR, uL, uR)]
    else:
        f = _hlld(L, R, fL, fR, uL, uR, torch.maximum(cL, cR), bs)
    f[5], f[8] = fb, fp
    return _back(f, D)


def _hlld(L, R, fL, fR, uL, uR, cf, bn):
    SL, SR = (torch.minimum(L[1], R[1]) - cf).clamp(max=0), (torch.maximum(L[1], R[1]) + cf).clamp(min=0)
    pt = [q[4] + 0.5 * (bn * bn + q[6] ** 2 + q[7] ** 2) for q in (L, R)]
    dS = [(S - q[1]) * q[0] for S, q in ((SL, L), (SR, R))]
    den = dS[1] - dS[0]
    SM = (dS[1] * R[1] - dS[0] * L[1] - pt[1] + pt[0]) / den
    ps = (dS[1] * pt[0] - dS[0] * pt[1] + dS[1] * dS[0] * (R[1] - L[1])) / den
    star, sq = [], []
    for q, u, S, d, p in ((L, uL, SL, dS[0], pt[0]), (R, uR, SR, dS[1], pt[1])):
        rs = (d / (S - SM)).clamp(min=1e-12)
        K = d * (S - SM) - bn * bn
        deg = K.abs() < (DTOL * bn * bn).clamp(min=1e-12)
        fac, r = bn * (SM - q[1]) / K, (d * (S - q[1]) - bn * bn) / K
        v, w = torch.where(deg, q[2], q[2] - q[6] * fac), torch.where(deg, q[3], q[3] - q[7] * fac)
        by, bz = torch.where(deg, q[6], q[6] * r), torch.where(deg, q[7], q[7] * r)
        vb, vbs = q[1] * bn + q[2] * q[6] + q[3] * q[7], SM * bn + v * by + w * bz
        star.append([rs, v, w, by, bz, ((S - q[1]) * u[4] - p * q[1] + ps * SM + bn * (vb - vbs)) / (S - SM), vbs])
        sq.append(rs.sqrt())
    sg = torch.where(bn >= 0, 1.0, -1.0).to(bn)
    inv = 1 / (sq[0] + sq[1])
    a, b = star
    v2, w2 = ((sq[0] * a[i] + sq[1] * b[i] + (b[i + 2] - a[i + 2]) * sg) * inv for i in (1, 2))
    by2, bz2 = ((sq[0] * b[i] + sq[1] * a[i] + sq[0] * sq[1] * (b[i - 2] - a[i - 2]) * sg) * inv for i in (3, 4))
    vb2 = SM * bn + v2 * by2 + w2 * bz2
    left, out = SM >= 0, []
    for q, f, u, S, k, s, sign in ((L, fL, uL, SL, a, sq[0], -1.0), (R, fR, uR, SR, b, sq[1], 1.0)):
        us = [k[0], k[0] * SM, k[0] * k[1], k[0] * k[2], k[5], bn, k[3], k[4]]
        u2 = [k[0], k[0] * SM, k[0] * v2, k[0] * w2, k[5] + sign * s * (k[6] - vb2) * sg, bn, by2, bz2]
        Ss = SM + sign * bn.abs() / s
        outer = Ss >= 0 if sign < 0 else Ss < 0
        out.append([torch.where(outer, f[i] + S * (us[i] - u[i]), f[i] + Ss * u2[i] - (Ss - S) * us[i] - S * u[i])
                    for i in range(8)])
    return [torch.where(left, x, y) for x, y in zip(*out)] + [torch.zeros_like(bn)]


def _ghost(n, lo, hi, bc):
    """Source indices of cells lo..hi-1 of an axis of n cells, and the wall's sign flips."""
    i = torch.arange(lo, hi, device=DEV)
    one = torch.ones(hi - lo, device=DEV, dtype=torch.float64)
    if bc == "periodic":
        return i % n, one
    if bc == "outflow":
        return i.clamp(0, n - 1), one
    out = (i < 0) | (i >= n)
    return torch.where(i < 0, -1 - i, torch.where(i >= n, 2 * n - 1 - i, i)).clamp(0, n - 1), torch.where(out, -one, one)


def _step64(U, c, dtdx, ch, decay, faces=None, q=None, vcorr=None):
    """One step of nine (nz, ny, nx) arrays; with faces also the new faces (constrained transport)."""
    nz, ny, nx = U[0].shape
    bcs = (c.get("bz", "periodic"), c.get("by", "periodic"), c.get("bx", "periodic"))
    recon, riemann = c.get("recon", "plm"), c.get("riemann", "hlld")
    iy, fy = _ghost(ny, -2, ny + 2, bcs[1])
    ix, fx = _ghost(nx, -2, nx + 2, bcs[2])
    new = [torch.empty_like(U[0], dtype=torch.float64) for _ in range(9)]
    ct = {k: torch.empty_like(new[0]) for k in ("m0", "m1", "m2", "xy", "xz", "yx", "yz", "zx", "zy", "ex", "ey", "ez")
          } if faces is not None else None
    step = max(1, min(nz, 6_000_000 // (ny * nx)))
    in1 = (slice(1, -1),) * 3
    for k0 in range(0, nz, step):
        k1 = min(nz, k0 + step)
        iz, fz = _ghost(nz, k0 - 2, k1 + 2, bcs[0])
        pad = lambda a: a[iz][:, iy][:, :, ix].double()  # noqa: E731
        P = [pad(a) for a in U]
        for comp, f in ((1, fx), (2, fy[:, None]), (3, fz[:, None, None])):
            P[comp], P[comp + 4] = P[comp] * f, P[comp + 4] * f
        P = _prim(P)

        def at(a, ax, o):
            return a[tuple(slice(1 + o, a.shape[d] - 1 + o) if d == ax else slice(1, -1) for d in range(3))]

        m0 = [a[in1] for a in P]
        off = [[_offsets(at(a, 2 - D, -1), at(a, 2 - D, 0), at(a, 2 - D, 1), recon) for a in P] for D in range(3)]
        acc = [0.0] * 9
        for D in range(3):
            hi = _back(_flux(_rot([a + o[1] for a, o in zip(m0, off[D])], D)), D)
            lo = _back(_flux(_rot([a + o[0] for a, o in zip(m0, off[D])], D)), D)
            acc = [a + (h - g) for a, h, g in zip(acc, hi, lo)]
        mh = _prim([a - 0.5 * dtdx * b for a, b in zip(_cons(m0), acc)])
        if q is not None:  # drag toward rest, integrated exactly over the half step
            fd, fp = math.exp(-0.5 * q), -math.expm1(-0.5 * q) / (0.5 * q)
            for i in (1, 2, 3):
                mh[i] = fd * m0[i] + fp * (mh[i] - m0[i])
                for D in range(3):
                    off[D][i] = tuple(fd * o for o in off[D][i])
        if vcorr is not None:
            for i in range(3):
                mh[1 + i] = mh[1 + i] + pad(vcorr[i])[in1]
        div = [0.0] * 9
        own = (slice(k0, k1), slice(None), slice(None))
        for D in range(3):
            ax = 2 - D
            cut = lambda a, s: a[tuple(s if d == ax else slice(1, -1) for d in range(3))]  # noqa: E731
            Lq = [cut(a + o[1], slice(0, -1)) for a, o in zip(mh, off[D])]
            Rq = [cut(a + o[0], slice(1, None)) for a, o in zip(mh, off[D])]
            bn = None
            if faces is not None:
                f = faces[D]
                bn = (f[torch.arange(k0, k1 + 1, device=DEV) % nz] if D == 2 else
                      torch.cat([f[k0:k1], f[k0:k1].narrow(ax, 0, 1)], ax)).double()
            F = _riemann(Lq, Rq, D, ch, riemann, bn)
            low = [a.narrow(ax, 0, a.shape[ax] - 1) for a in F]
            div = [d + (a - b.narrow(ax, 1, b.shape[ax] - 1)) for d, a, b in zip(div, low, F)]
            if ct is not None:
                ct["m%d" % D][own] = low[0]
                for e, name in enumerate("xyz"):
                    if e != D:
                        ct["xyz"[D] + name][own] = low[5 + e]
            del F, Lq, Rq
        u0 = [a[k0:k1].double() for a in U]
        t = [a + dtdx * d for a, d in zip(u0, div)]
        if q is not None:
            e, p1 = math.exp(-q), -math.expm1(-q) / q
            em1, em2 = -math.expm1(-q), -math.expm1(-2 * q)
            w = [u0[i] / u0[0] for i in (1, 2, 3)]
            dv = [t[i] / t[0] - a for i, a in zip((1, 2, 3), w)]
            t[4] = t[4] - t[0] * (0.5 * em2 * sum(a * a for a in w) + em1 * em1 / q * sum(a * b for a, b in zip(w, dv)) +
                                  (q - 2 * em1 + 0.5 * em2) / (q * q) * sum(b * b for b in dv))
            for i in range(3):
                t[1 + i] = t[0] * (e * w[i] + p1 * dv[i])
        t[8] = t[8] * decay if faces is None else torch.zeros_like(t[8])
        for a, b in zip(new, t):
            a[own] = b
        if ct is not None:
            b0, v = [a[1:-1, 1:-1, 1:-1] for a in m0[5:8]], [a[1:-1, 1:-1, 1:-1] for a in mh[1:4]]
            ct["ex"][own], ct["ey"][own] = v[2] * b0[1] - v[1] * b0[2], v[0] * b0[2] - v[2] * b0[0]
            ct["ez"][own] = v[1] * b0[0] - v[0] * b0[1]
        del P, m0, off, mh, acc, div, t, u0
    if faces is None:
        return new
    f = _ct_faces(ct, [a.double() for a in faces], dtdx)
    for d in range(3):
        new[5 + d] = 0.5 * (f[d] + _up(f[d], 2 - d))
    return new, f


def _ct_faces(w, f, dtdx):
    """Contact-upwinded edge EMFs and the curl of them on the faces."""
    def edge(Ea, Eb, mA, mB, Er, a, b):  # a: the axis along which Ea and mA step, b: the other
        def up(m, lo, hi):
            return torch.where(m > 0, lo, torch.where(m < 0, hi, 0.5 * (lo + hi)))
        Eam, Ebm, mAm, mBm = _dn(Ea, a), _dn(Eb, b), _dn(mA, a), _dn(mB, b)
        Em0, E0m = _dn(Er, b), _dn(Er, a)
        Emm = _dn(Em0, a)
        A = up(mAm, Ebm - Emm, Eb - E0m) - up(mA, Em0 - Ebm, Er - Eb)
        B = up(mBm, Eam - Emm, Ea - Em0) - up(mB, E0m - Eam, Er - Ea)
        return 0.25 * ((Ea + Eam + Eb + Ebm) + A + B)
    ez = edge(-w["xy"], w["yx"], w["m0"], w["m1"], w["ez"], 1, 2)
    ex = edge(-w["yz"], w["zy"], w["m1"], w["m2"], w["ex"], 0, 1)
    ey = edge(-w["zx"], w["xz"], w["m2"], w["m0"], w["ey"], 2, 0)
    return [f[0] - dtdx * ((_up(ez, 1) - ez) - (_up(ey, 0) - ey)), f[1] - dtdx * ((_up(ex, 0) - ex) - (_up(ez, 2) - ez)),
            f[2] - dtdx * ((_up(ey, 2) - ey) - (_up(ex, 1) - ex))]


def _terminal_velocity(U, B, dx):
    rho = U[0]
    B = [b.double() for b in B]
    F = []
    half = 0.5 * sum(b * b for b in B)
    for i in range(3):
        F.append(sum(_up(T, 2 - d) - _dn(T, 2 - d) for d, T in
                     ((d, B[i] * B[d] - (half if i == d else 0.0)) for d in range(3))) / (2 * dx))
    return [(F[d] - 0.2 * (_up(rho, 2 - d) - _dn(rho, 2 - d)) / (2 * dx)) / (rho * 4.0) for d in range(3)]


def _terminal64(U, faces, c, dt):
    dx = _dx(c)
    U = [u.double() for u in U]
    B0 = U[5:8]

    def emf(B):
        v = _terminal_velocity(U, B, dx)
        return [v[1] * B[2] - v[2] * B[1], v[2] * B[0] - v[0] * B[2], v[0] * B[1] - v[1] * B[0]]

    vmax = float(sum(v.square() for v in _terminal_velocity(U, B0, dx)).max().sqrt())
    order = c["order"]
    eta = 0.05 / 12 * vmax * dx ** 3 if order == 4 else 0.05 * vmax * dx

    def lap(a):
        return (sum(_up(a, x) + _dn(a, x) for x in range(3)) - 6 * a) / (dx * dx)

    def rate(B, A):
        e = emf(B)
        if faces is None:
            d = lambda a, x: (_up(a, x) - _dn(a, x)) / (2 * dx)  # noqa: E731
        else:
            av = lambda a, x, y: 0.25 * (a + _dn(a, x) + _dn(a, y) + _dn(_dn(a, x), y))  # noqa: E731
            e = [av(e[0], 0, 1), av(e[1], 0, 2), av(e[2], 1, 2)]
            d = lambda a, x: (_up(a, x) - a) / dx  # noqa: E731
        curl = [d(e[2], 1) - d(e[1], 0), d(e[0], 0) - d(e[2], 2), d(e[1], 2) - d(e[0], 1)]
        return [r - eta * lap(lap(a)) if order == 4 else r + eta * lap(a) for r, a in zip(curl, A)]

    A = [f.double() for f in faces] if faces is not None else B0
    avg = (lambda f: [0.5 * (a + _up(a, 2 - d)) for d, a in enumerate(f)]) if faces is not None else (lambda f: f)
    p = [a + dt * r for a, r in zip(A, rate(B0, A))]
    n = [0.5 * (a + b + dt * r) for a, b, r in zip(A, p, rate(avg(p), p))]
    B = avg(n)
    E = U[4] + 0.5 * (sum(b * b for b in B) - sum(b * b for b in B0))
    flat = [a.reshape(-1) for a in (U[0], E, *B)]
    return flat + ([torch.cat([a.reshape(-1) for a in n])] if faces is not None else [])


def _evolve64(U, faces, c, dx, tfinal=None, steps=None):
    """CFL-limited steps to tfinal, or a number of them."""
    t, n = 0.0, 0
    while (t < tfinal * (1 - 1e-9)) if steps is None else n < steps:
        smax = max(_wavespeed([u[k:k + 32].double() for u in U]) for k in range(0, U[0].shape[0], 32))
        dt = CFL * dx / smax
        if steps is None:
            dt = min(dt, tfinal - t)
        if faces is None:
            U = _step64(U, c, dt / dx, smax, math.exp(-CR * smax * dt / dx))
        else:
            U, faces = _step64(U, c, dt / dx, 0.0, 1.0, faces)
        t, n = t + dt, n + 1
    return U, faces, n


def exact(case, seed):
    flat = lambda v: torch.cat([a.reshape(-1) for a in v])  # noqa: E731
    if case["kind"] == "batch":
        fields, faces = [], []
        for i, b in enumerate(_mix(case)):
            U, f = _fields((b["n"],) * 3, seed * 1000 + i, b["solver"], b["beta"], b["index"], b["kc"])
            U, f, _ = _evolve64(U, f, {}, _f32(1.0 / b["n"]), steps=2)
            fields += U
            faces += [flat(f)] if f is not None else []
        return [flat(fields), flat(faces) if faces else torch.zeros(0, dtype=torch.float64, device=DEV)]
    U, faces, par = _inputs(case, seed)
    if case["kind"] == "terminal":
        return _terminal64(U, faces, case, par["dt"])
    if case["kind"] == "ledger":
        dx = _dx(case)
        dV = _f32(np.float32(dx) * np.float32(dx) * np.float32(dx))
        div = sum(_up(b, 2 - d) - _dn(b, 2 - d) for d, b in enumerate(u.double() for u in U[5:8])) / (2 * dx)
        return [np.array([float(u.double().sum()) * dV for u in U[:8]]), np.float64(div.abs().max().item())]
    if case["kind"] == "evolve":
        U, faces, n = _evolve64(U, faces, case, _dx(case), 3.5 * par["dt"])
        return [u.reshape(-1) for u in U] + ([flat(faces)] if faces is not None else []) + [n]
    dtdx = par["dt"] / _dx(case)
    if case["kind"] in ("drag", "rad"):
        vc = _corrections(case, seed) if case["kind"] == "rad" else None
        new = _step64(U, case, dtdx, par["ch"], par["decay"], q=_f32(0.05), vcorr=vc)
        extra = [(new[0] - U[0].double()).reshape(-1)] if vc is not None else []
        return [u.reshape(-1) for u in new] + extra
    if faces is not None:
        new, f = _step64(U, case, dtdx, 0.0, 1.0, faces)
        return [u.reshape(-1) for u in new] + [flat(f)]
    return [u.reshape(-1) for u in _step64(U, case, dtdx, par["ch"], par["decay"])]
