"""What a user of the solver has it do, as measurable cases.

Every case is one pass of a user's program through the public interface
(`hydrocode_astro1_b200`): rewind a context to the state it keeps in hand and
take a few time steps, step a host array as an embedding C code does, or train
the learned warm start.  The set-ups are the repository's own configurations
(`problems.py`: Sod tube, n=1 polytrope, cold collapse, stellar explosion in
the centred and the octant layout, close binary) and a generic subsonic flow,
made on the GPU from a seed, with the explosion's log-normal density noise on
every one of them so that another seed is another realisation.

A self-gravitating run solves each step's Poisson problem from the previous
step's potential.  `prepare` therefore hands the context the converged
potential of its first state (a direct sine-transform solve of the discrete
equation, as a restart file would hold it), not a cold start; within a pass,
step k's solve starts from step k-1's potential, and the first solve of a
repeated pass from the potential the pass before it ended with -- except with
the learned start, which is trained on a run's successive residuals: there
`prepare` takes a few steps, keeps the state and the potential they reach, and
a pass rewinds both.

The state crosses to and from the context on the device, in the context's
precision; a double-precision run with gravity also returns its potential.
The mixed-precision runs return the FP32 state: their potential is defined
only to the solver's tolerance.
"""
from __future__ import annotations

import ctypes
import functools
import math
import os

import numpy as np
import torch

import hydrocode_astro1_b200 as hc
from hydrocode_astro1_b200 import problems

RHO_FLOOR, P_FLOOR = 1.0e-5, 1.0e-6
OUT = "222222"          # outflow on every face (xmin xmax ymin ymax zmin zmax)
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(hc.__file__)), "data", "unet_stellar_explosion_256.bin")


def listed():
    return [
        # the embedding C program: a small self-gravitating star on a host array,
        # four calls of one step with the drop-in's default settings -- all latency
        dict(name="host_step_20x18x22", kind="host", problem="polytrope", nx=20, ny=18, nz=22, fp32=False, lmax=0,
             sequential=True, tol=1e-6, bc=OUT, steps=4),
        # the Sod tube, the plain double-precision method without gravity
        dict(name="sod_64_fp64", kind="run", problem="sod", nx=64, ny=64, nz=64, fp32=False, lmax=-1,
             sequential=False, tol=0.0, bc=OUT, steps=10),
        # the polytrope with the drop-in's defaults: the reference's own boundary
        # expansion and summation order
        dict(name="polytrope_128_fp64", kind="run", problem="polytrope", nx=128, ny=128, nz=128, fp32=False, lmax=0,
             sequential=True, tol=1e-8, bc=OUT, steps=2),
        # a ragged grid with mirror faces (the octant layout), double precision
        dict(name="octant_90x101x97_fp64", kind="run", problem="octant", nx=90, ny=101, nz=97, fp32=False, lmax=0,
             sequential=False, tol=1e-6, bc="121212", steps=3),
        # second-order reconstruction
        dict(name="plm_128_fp64", kind="plm", problem="flow", nx=128, ny=128, nz=128, fp32=False, lmax=-1,
             sequential=False, tol=0.0, bc="000000", steps=4),
        # single-precision gas dynamics alone at the benchmark's size
        dict(name="flow_256_fp32", kind="run", problem="flow", nx=256, ny=256, nz=256, fp32=True, lmax=-1,
             sequential=False, tol=0.0, bc="002222", steps=10),
        # cold collapse, mixed precision
        dict(name="collapse_192_mixed", kind="run", problem="collapse", nx=192, ny=192, nz=192, fp32=True, lmax=8,
             sequential=False, tol=1e-8, bc=OUT, steps=2),
        # the benchmark's three arms: mixed precision from the previous potential,
        # with the learned start, and double precision
        dict(name="explosion_256_mixed", kind="run", problem="explosion", nx=256, ny=256, nz=256, fp32=True, lmax=8,
             sequential=False, tol=1e-8, bc=OUT, steps=3),
        dict(name="explosion_256_learned", kind="learned", problem="explosion", nx=256, ny=256, nz=256, fp32=True,
             lmax=8, sequential=False, tol=1e-8, bc=OUT, lead=4, steps=5),
        dict(name="explosion_256_fp64", kind="run", problem="explosion", nx=256, ny=256, nz=256, fp32=False, lmax=8,
             sequential=False, tol=1e-8, bc=OUT, steps=2),
        # the largest grid: the close binary at the drop-in's default tolerance
        dict(name="binary_512_mixed", kind="run", problem="binary", nx=512, ny=512, nz=512, fp32=True, lmax=12,
             sequential=False, tol=1e-6, bc=OUT, steps=3),
        # training the learned start at the benchmark's network size
        dict(name="train_256", kind="train", problem="explosion", nx=256, ny=256, nz=256, fp32=True, lmax=8,
             sequential=False, tol=1e-6, bc=OUT, steps=6),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "gas64", "gas32", "plm", "grav64", "grav64", "mixed", "mixed", "mixed", "learned", "train"])
    tri = lambda lo, hi: [_spread(rng, lo, hi) for _ in range(3)]                      # noqa: E731
    near = lambda n: [max(8, int(round(n * rng.uniform(0.8, 1.2)))) for _ in range(3)]   # noqa: E731
    c = dict(kind="run", problem="flow", fp32=False, lmax=-1, sequential=False, tol=0.0, bc=OUT, steps=4)
    if kind == "host":
        dims = tri(12, 64)
        c.update(kind="host", problem="polytrope", lmax=0, sequential=True, tol=1e-6, steps=rng.randint(2, 5))
    elif kind in ("gas64", "gas32"):
        dims = tri(16, 256)
        c.update(fp32=kind == "gas32", problem=rng.choice(["sod", "flow"]), bc=rng.choice([OUT, "000000", "121212", "110022"]))
    elif kind == "plm":
        dims = tri(16, 160)
        c.update(kind="plm", bc=rng.choice([OUT, "000000", "121212"]))
    elif kind == "grav64":
        dims = near(_spread(rng, 24, 160))
        c.update(problem=rng.choice(["polytrope", "collapse", "explosion"]), lmax=rng.choice([0, 0, 4, 8]),
                 tol=rng.choice([1e-6, 1e-8]), steps=2)
        c.update(sequential=c["lmax"] == 0 and rng.random() < 0.7)
    elif kind == "mixed":
        n = _spread(rng, 32, 256)
        dims = [n, n, n] if rng.random() < 0.5 else near(n)
        c.update(problem=rng.choice(["polytrope", "collapse", "explosion", "binary"]), lmax=rng.choice([0, 4, 8, 12]),
                 fp32=True, tol=rng.choice([1e-6, 1e-8]), steps=2)
    else:
        n = 32 * rng.randint(3, 8)
        dims = [n, n, 32 * rng.randint(3, 8)] if rng.random() < 0.3 else [n, n, n]
        c.update(kind=kind, problem="explosion", lmax=8, fp32=True, tol=1e-8, steps=3)
        if kind == "train":
            c.update(tol=1e-6, steps=rng.randint(3, 10))
        else:
            c.update(lead=rng.randint(2, 6))
    c.update(nx=dims[0], ny=dims[1], nz=dims[2])
    return c


# ---------------------------------------------------------------- set-ups
BOX = {"sod": (0.0, 1.0), "flow": (0.0, 1.0), "polytrope": (0.0, 1.0), "collapse": (-2.0, 2.0),
       "explosion": (-0.75, 0.75), "octant": (0.0, 1.5), "binary": (-1.0, 1.0)}
GAMMA = {"sod": 1.4, "flow": 1.4, "polytrope": 2.0, "collapse": 5.0 / 3.0, "explosion": 5.0 / 3.0,
         "octant": 5.0 / 3.0, "binary": 2.0}


@functools.lru_cache(maxsize=1)
def _star():
    return problems.polytrope_profile(3, 1.0, 0.4)


def _shape(c):
    return c["nx"], c["ny"], c["nz"]


def _spacing(c):
    lo, hi = BOX[c["problem"]]
    return [(hi - lo) / n for n in _shape(c)]


def _axes(c):
    lo, _ = BOX[c["problem"]]
    d = _spacing(c)
    ax = [lo + (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) * d[a] for a, n in enumerate(_shape(c))]
    return ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]


def _interp(x, xp, fp):
    xp, fp = (torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device="cuda") for v in (xp, fp))
    k = torch.clamp(torch.searchsorted(xp, x.contiguous()), 1, xp.numel() - 1)
    w = torch.clamp((x - xp[k - 1]) / (xp[k] - xp[k - 1]), 0.0, 1.0)
    return fp[k - 1] * (1.0 - w) + fp[k] * w


def _primitives(c, seed):
    """rho, u, v, w, p of the first state, FP64 on the GPU."""
    shape, gam, prob = _shape(c), GAMMA[c["problem"]], c["problem"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    X, Y, Z = _axes(c)
    zero = torch.zeros(shape, dtype=torch.float64, device="cuda")
    vel = [zero, zero, zero]
    noise = torch.exp(0.01 * torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda"))
    if prob == "sod":
        left = (X < 0.5).expand(shape)
        rho = torch.where(left, 1.0, 0.125) * noise
        p = torch.where(left, 1.0, 0.1) + zero
    elif prob == "flow":
        ph = torch.rand(5, 3, generator=gen, dtype=torch.float64, device="cuda") * 2.0 * math.pi
        wave = lambda q: (torch.sin(2 * math.pi * X + ph[q, 0]) * torch.cos(2 * math.pi * Y + ph[q, 1])
                          * torch.cos(2 * math.pi * Z + ph[q, 2]))  # noqa: E731
        rho = (1.0 + 0.3 * wave(0)) * noise
        vel = [0.4 * wave(q) for q in (1, 2, 3)]
        p = 1.0 + 0.2 * wave(4)
    elif prob == "polytrope":
        r = torch.sqrt((X - 0.5) ** 2 + (Y - 0.5) ** 2 + (Z - 0.5) ** 2)
        rho_c = math.pi / (4.0 * 0.35 ** 3)
        rho = torch.clamp(torch.where(r < 0.35, rho_c * torch.sinc(r / 0.35), 0.0), min=1e-6 * rho_c) * noise
        p = 2.0 * 0.35 ** 2 / math.pi * rho * rho
    elif prob == "collapse":
        r = torch.sqrt(X * X + Y * Y + Z * Z)
        rs = torch.clamp(r, min=2.0 * max(_spacing(c)))
        inside = r < 1.0
        rho = torch.where(inside, 1.0 / (2.0 * math.pi * rs), 1e-5)
        rho = torch.where(inside, rho / (rho[inside].sum() * math.prod(_spacing(c))), rho) * noise
        p = (gam - 1.0) * rho * 0.05
    elif prob == "binary":
        rho, p, vy = zero + RHO_FLOOR, zero + P_FLOOR, zero.clone()
        v_orb = math.sqrt(0.8 / 0.5)
        for xc, M, v in ((-0.5 * 0.3 / 0.8, 0.5, v_orb * 0.3 / 0.8), (0.5 * 0.5 / 0.8, 0.3, -v_orb * 0.5 / 0.8)):
            r = torch.sqrt((X - xc) ** 2 + Y * Y + Z * Z)
            s = torch.where(r < 0.15, math.pi * M / (4.0 * 0.15 ** 3) * torch.sinc(r / 0.15), 0.0) * noise
            rho = torch.where(r < 0.15, torch.clamp(s, min=RHO_FLOOR), rho)
            p = torch.where(r < 0.15, torch.clamp(2.0 * 0.15 ** 2 / math.pi * s * s, min=P_FLOOR), p)
            vy = torch.where(r < 0.15, v, vy)
        vel = [zero, vy, zero]
    else:   # explosion (centred) and octant
        r_tab, rho_tab, u_tab = _star()
        r = torch.sqrt(X * X + Y * Y + Z * Z)
        rho, u = _interp(r, r_tab, rho_tab), _interp(r, r_tab, u_tab)
        out = r >= 0.4
        rho, u = torch.where(out, 1e-6, rho) * noise, torch.where(out, 1e-6, u)
        d = _spacing(c)
        hot = r < max(0.02 * 0.4, 1.01 * math.sqrt(sum(x * x for x in d)))
        u = torch.where(hot, u + 1.0 / (hot.sum() * math.prod(d)) / rho, u)
        p = rho * u * (gam - 1.0)
    return [rho] + vel + [p]


def _to_cons(w, gam):
    rho, u, v, s, p = w
    return torch.stack([rho, rho * u, rho * v, rho * s, p / (gam - 1.0) + 0.5 * rho * (u * u + v * v + s * s)])


def _first_state(c, seed):
    return _to_cons(_primitives(c, seed), GAMMA[c["problem"]])


# ---------------------------------------------------------------- prepare / run
def prepare(case, seed):
    c = dict(case)
    gravity = c["lmax"] >= 0
    lo, hi = BOX[c["problem"]]
    q = _first_state(c, seed)
    s = hc.HydroSolver3D(_shape(c), lo=(lo,) * 3, hi=(hi,) * 3, gamma=GAMMA[c["problem"]], cfl=0.4,
                         G=1.0 if gravity else 0.0, bc=[int(b) for b in c["bc"]], lmax=max(0, c["lmax"]),
                         tol=c["tol"] if gravity else 1e-6, max_iter=20000,
                         precision=hc.FP32 if c["fp32"] else hc.FP64,
                         moment_order=hc.MOMENTS_SEQUENTIAL if c["sequential"] else hc.MOMENTS_TREE,
                         recon=1 if c["kind"] == "plm" else 0,
                         warm_start=hc.WARM_UNET if c["kind"] == "learned" else hc.WARM_PREVIOUS)
    st = {"case": c, "solver": s}
    if gravity:
        phi = np.ascontiguousarray(_potential(c, q[0]).cpu().numpy())
        s.set_phi(phi)
    if c["kind"] == "host":
        st["U0"] = np.ascontiguousarray(q.permute(1, 2, 3, 0).cpu().numpy())
        st["U"] = np.empty_like(st["U0"])
        return st
    st["first"] = q.to(torch.float32 if c["fp32"] else torch.float64).contiguous()
    st["out"] = torch.empty_like(st["first"])
    if gravity and not c["fp32"]:
        st["phi"] = torch.empty(_shape(c), dtype=torch.float64, pin_memory=True)
    torch.cuda.synchronize()
    s.copy_planes(0, c["nx"], st["first"].data_ptr(), True)
    if c["kind"] == "learned":
        s.unet_load_file(WEIGHTS)
        s.step(c["lead"])
        s.copy_planes(0, c["nx"], st["first"].data_ptr(), False)
        st["phi0"] = torch.from_numpy(s.phi()).pin_memory()
    st["speed"] = s.signal_speed()
    if c["kind"] == "train":   # two recorded solves to train on, and the weights to start from
        s.unet_init(int(seed) % (1 << 31))
        s.unet_collect(2)
        s.step(3)
        st["weights"], st["kscale"] = s.unet_params()
    return st


def _doubles(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _ok(rc):
    if rc != hc.HC_OK:
        raise RuntimeError(hc.last_error())


def run(state):
    c, s = state["case"], state["solver"]
    if c["kind"] == "host":
        state["U"][...] = state["U0"]
        dts = [s.step_host(state["U"]) for _ in range(c["steps"])]
        return {"U": state["U"], "dt": dts}
    if c["kind"] == "train":
        s.unet_load(state["weights"], state["kscale"])
        loss = s.unet_train(c["steps"], 1e-3, 1)
        return {"weights": s.unet_params()[0], "loss": np.float32(loss)}
    s.copy_planes(0, c["nx"], state["first"].data_ptr(), True)
    s.set_signal_speed(state["speed"])
    if "phi0" in state:
        _ok(s.L.hc_set_phi(s.h, _doubles(state["phi0"])))
    dts = s.step(c["steps"])
    s.copy_planes(0, c["nx"], state["out"].data_ptr(), False)
    got = {"state": state["out"], "dt": dts.astype(np.float32) if c["fp32"] else dts}
    if "phi" in state:
        _ok(s.L.hc_get_phi(s.h, _doubles(state["phi"])))
        got["phi"] = state["phi"]
    return got


def work(case):
    """Each field read once and written once per step; the relaxation sweeps
    (about 4 n of them for the solves of these set-ups) as arithmetic only,
    since nothing but their first and last touch of a field has to leave the
    chip."""
    c = dict(case)
    n, w = math.prod(_shape(c)), 4 if c["fp32"] else 8
    if c["kind"] == "train":
        vox, levels = n // 8, sum(8.0 ** -k for k in range(5)) + sum(8.0 ** -k for k in range(5))
        flops = 2 * 27 * 16 * 16 * vox * levels
        return {"bytes": c["steps"] * vox * (2 * 4 + 4 * 32 * levels), "flops": c["steps"] * 3 * flops}
    gravity = c["lmax"] >= 0
    per = 10 * w + (16 if gravity else 0)
    flops = (900 if c["kind"] == "plm" else 450) + (4 * max(_shape(c)) * 13 if gravity else 0)
    crossing = 80 * n * c["steps"] if c["kind"] == "host" else 0
    return {"bytes": c["steps"] * n * per + crossing, "flops": c["steps"] * n * flops}


# ---------------------------------------------------------------- 64-bit restatement
def _harmonic_boundary(c, rho, pts):
    """Exterior potential at pts (three broadcastable tensors) of the cells
    with rho > 0: monopole and Cartesian quadrupole about the centre of mass
    (lmax 0), or solid harmonics to degree lmax."""
    X, Y, Z = _axes(c)
    dm = torch.clamp(rho, min=0.0) * math.prod(_spacing(c))
    M = dm.sum()
    com = [(dm * A).sum() / M for A in (X, Y, Z)]
    A = [X - com[0], Y - com[1], Z - com[2]]
    B = [pts[a] - com[a] for a in range(3)]
    R2 = B[0] ** 2 + B[1] ** 2 + B[2] ** 2
    R = torch.sqrt(R2)
    if c["lmax"] == 0:
        r2 = A[0] ** 2 + A[1] ** 2 + A[2] ** 2
        Qr = 0.0
        for a in range(3):
            for b in range(3):
                Qr = Qr + (dm * (3.0 * A[a] * A[b] - (r2 if a == b else 0.0))).sum() * B[a] * B[b]
        return -M / R - Qr / (2.0 * R ** 5)
    pot = 0.0
    for m in range(c["lmax"] + 1):
        src, dst = _degrees(A, m, c["lmax"]), _degrees(B, m, c["lmax"])
        for l, ((sr, si), (tr, ti)) in enumerate(zip(src, dst), start=m):
            norm = (1.0 if m == 0 else 2.0) * math.factorial(l - m) / math.factorial(l + m)
            term = (dm * sr).sum() * tr + (dm * si).sum() * ti
            pot = pot - norm * term / R ** (2 * l + 1)
    return pot


def _degrees(P, m, lmax):
    """r^l P_l^m e^{i m phi} for l = m .. lmax, as (real, imaginary)."""
    x, y, z = P
    z = z + 0.0 * (x + y)
    r2 = x * x + y * y + z * z
    qr, qi = torch.ones_like(z), torch.zeros_like(z)
    for k in range(1, m + 1):
        qr, qi = (2 * k - 1) * (x * qr - y * qi), (2 * k - 1) * (x * qi + y * qr)
    got = [(qr, qi)]
    for l in range(m + 1, lmax + 1):
        (pr, pi), (or_, oi) = got[-1], got[-2] if l > m + 1 else (0.0, 0.0)
        got.append((((2 * l - 1) * z * pr - (l + m - 1) * r2 * or_) / (l - m),
                    ((2 * l - 1) * z * pi - (l + m - 1) * r2 * oi) / (l - m)))
    return got


def _potential(c, rho):
    """The discrete Poisson equation (7-point, Dirichlet values from the
    multipole expansion of rho on the outermost cells) solved directly by sine
    transforms of its interior."""
    shape, d = _shape(c), _spacing(c)
    ax = _axes(c)
    phi = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for a in range(3):
        for side in (0, shape[a] - 1):
            at = [slice(None)] * 3
            at[a] = slice(side, side + 1)
            pts = [v[tuple(slice(None) if v.shape[b] == 1 else at[b] for b in range(3))] for v in ax]
            phi[tuple(at)] = _harmonic_boundary(c, rho, pts)
    f = 4.0 * math.pi * rho[1:-1, 1:-1, 1:-1]
    for a in range(3):
        lead = [slice(1, -1)] * 3
        for side, row in ((0, 0), (-1, -1)):
            at = list(lead)
            at[a] = side
            to = [slice(None)] * 3
            to[a] = row
            f[tuple(to)] -= phi[tuple(at)] / d[a] ** 2
    lam = 0.0
    for a in range(3):
        n = shape[a] - 2
        k = torch.arange(1, n + 1, dtype=torch.float64, device="cuda")
        S = torch.sin(math.pi / (n + 1) * k[:, None] * k[None, :]) * math.sqrt(2.0 / (n + 1))
        f = torch.tensordot(f, S, dims=([a], [0])).movedim(-1, a)
        e = (2.0 * torch.cos(math.pi * k / (n + 1)) - 2.0) / d[a] ** 2
        lam = lam + e.reshape([n if b == a else 1 for b in range(3)])
    f = f / lam
    for a in range(3):
        n = shape[a] - 2
        k = torch.arange(1, n + 1, dtype=torch.float64, device="cuda")
        S = torch.sin(math.pi / (n + 1) * k[:, None] * k[None, :]) * math.sqrt(2.0 / (n + 1))
        f = torch.tensordot(f, S, dims=([a], [0])).movedim(-1, a)
    phi[1:-1, 1:-1, 1:-1] = f
    return phi


def _prims(q, gam):
    rho = torch.clamp(q[0], min=RHO_FLOOR)
    u, v, w = q[1] / rho, q[2] / rho, q[3] / rho
    p = torch.clamp((gam - 1.0) * (q[4] - 0.5 * rho * (u * u + v * v + w * w)), min=P_FLOOR)
    return [rho, u, v, w, p]


def _speed(q, gam):
    w = _prims(q, gam)
    return float((torch.stack([w[1].abs(), w[2].abs(), w[3].abs()]).amax(0) + torch.sqrt(gam * w[4] / w[0])).max())


def _hllc(qL, wL, qR, wR, a, gam):
    """HLLC flux along axis a between states given as conserved and primitive."""
    cL, cR = torch.sqrt(gam * wL[4] / wL[0]), torch.sqrt(gam * wR[4] / wR[0])
    uL, uR = wL[1 + a], wR[1 + a]
    sL, sR = torch.minimum(uL - cL, uR - cR), torch.maximum(uL + cL, uR + cR)
    aL, aR = wL[0] * (sL - uL), wR[0] * (sR - uR)
    ss = (wR[4] - wL[4] + aL * uL - aR * uR) / (aL - aR)
    left = (sL >= 0) | ((sR > 0) & (ss >= 0))
    star = (sL < 0) & (sR > 0)
    q = [torch.where(left, qL[v], qR[v]) for v in range(5)]
    w = [torch.where(left, wL[v], wR[v]) for v in range(5)]
    sK = torch.where(left, sL, sR)
    un = w[1 + a]
    f = [q[v] * un for v in range(5)]
    f[0] = q[1 + a]
    f[1 + a] = f[1 + a] + w[4]
    f[4] = (q[4] + w[4]) * un
    rs = w[0] * (sK - un) / (sK - ss)
    us = [rs, rs * w[1], rs * w[2], rs * w[3],
          rs * (q[4] / w[0] + (ss - un) * (ss + w[4] / (w[0] * (sK - un))))]
    us[1 + a] = rs * ss
    return [torch.where(star, f[v] + sK * (us[v] - q[v]), f[v]) for v in range(5)]


def _cut(t, a, lo, hi):
    at = [slice(None)] * t.dim()
    at[a + t.dim() - 3] = slice(lo, hi)
    return t[tuple(at)]


def _half_step(w, c, dt, gam):
    """MUSCL-Hancock: half-advanced primitives and limited slopes."""
    d, sl = _spacing(c), []
    for a in range(3):
        n = _shape(c)[a]
        dw = torch.zeros_like(w)
        lo, hi = _cut(w, a, 1, n - 1) - _cut(w, a, 0, n - 2), _cut(w, a, 2, n) - _cut(w, a, 1, n - 1)
        _cut(dw, a, 1, n - 1).copy_(torch.where(lo * hi <= 0, 0.0, torch.where(lo.abs() < hi.abs(), lo, hi)))
        sl.append(dw)
    ws = w.clone()
    for a in range(3):
        un, dw = w[1 + a], sl[a]
        t = un * dw
        t[0] += w[0] * dw[1 + a]
        t[1 + a] += dw[4] / w[0]
        t[4] += gam * w[4] * dw[1 + a]
        ws = ws - 0.5 * dt / d[a] * t
    ok = (ws[0] > 0) & (ws[4] > 0)
    for a in range(3):
        for sgn in (0.5, -0.5):
            ok &= (ws[0] + sgn * sl[a][0] > 0) & (ws[4] + sgn * sl[a][4] > 0)
    return torch.where(ok, ws, w), [torch.where(ok, s, 0.0) for s in sl]


def _advance(q, c, smax, phi):
    """One unsplit Godunov step; returns the new state and its dt."""
    gam, d, shape = GAMMA[c["problem"]], _spacing(c), _shape(c)
    dt = 0.4 * min(d) / max(smax, 1e-10)
    w = torch.stack(_prims(q, gam))
    if c["kind"] == "plm":
        ws, sl = _half_step(w, c, dt, gam)
    new = q.clone()
    inner = (slice(1, -1),) * 3
    for a in range(3):
        n = shape[a]
        if c["kind"] == "plm":
            wL, wR = _cut(ws + 0.5 * sl[a], a, 0, n - 1), _cut(ws - 0.5 * sl[a], a, 1, n)
            qL, qR = _to_cons(wL, gam), _to_cons(wR, gam)
            wL, wR = _prims(qL, gam), _prims(qR, gam)
        else:
            wL, wR = _cut(w, a, 0, n - 1), _cut(w, a, 1, n)
            qL, qR = _cut(q, a, 0, n - 1), _cut(q, a, 1, n)
        for b in range(3):
            if b != a:
                m = shape[b]
                qL, qR = _cut(qL, b, 1, m - 1), _cut(qR, b, 1, m - 1)
                if torch.is_tensor(wL):
                    wL, wR = _cut(wL, b, 1, m - 1), _cut(wR, b, 1, m - 1)
                else:
                    wL, wR = [_cut(x, b, 1, m - 1) for x in wL], [_cut(x, b, 1, m - 1) for x in wR]
        f = _hllc(qL, wL, qR, wR, a, gam)
        for v in range(5):
            new[v][inner] -= dt / d[a] * (_cut(f[v], a, 1, n - 1) - _cut(f[v], a, 0, n - 2))
    new[(slice(None),) + inner] = _to_cons(_prims(new[(slice(None),) + inner], gam), gam)
    if phi is not None:
        g = []
        for a in range(3):
            n = shape[a]
            gi = -(_cut(phi, a, 2, n) - _cut(phi, a, 0, n - 2)) / (2.0 * d[a])
            for b in range(3):
                if b != a:
                    gi = _cut(gi, b, 1, shape[b] - 1)
            g.append(torch.nn.functional.pad(gi[None, None], (1,) * 6, mode="replicate")[0, 0])
        old = new.clone()
        new[4] += dt * (old[1] * g[0] + old[2] * g[1] + old[3] * g[2])
        for a in range(3):
            new[1 + a] += dt * old[0] * g[a]
    bc = [int(b) for b in c["bc"]]
    for a in range(3):
        if bc[2 * a] == 0 and bc[2 * a + 1] == 0:
            _cut(new, a, 0, 1).copy_(_cut(new, a, shape[a] - 1, shape[a]).clone())
    for a in range(3):
        n = shape[a]
        for side, b, i in ((0, 0, 1), (1, n - 1, n - 2)):
            edge = _cut(new, a, b, b + 1)
            if bc[2 * a + side] == 1:
                we = _prims(edge.clone(), gam)
                we[1 + a] = -we[1 + a]
                edge.copy_(_to_cons(we, gam))
            elif bc[2 * a + side] == 2:
                edge.copy_(_cut(new, a, i, i + 1).clone())
    return new, dt


def exact(case, seed):
    """The steps of a pass in 64 bits: the gas update above, the Poisson
    equation solved directly.  A trained network has no such value."""
    c = dict(case)
    if c["kind"] == "train":
        return None
    q = _first_state(c, seed)
    if c["fp32"]:
        q = q.float().double()
    gam, dts, phi = GAMMA[c["problem"]], [], None
    for _ in range(c.get("lead", 0) + c["steps"]):
        if c["lmax"] >= 0:
            phi = _potential(c, q[0])
        q, dt = _advance(q, c, _speed(q, gam), phi)
        dts.append(dt)
    if c["kind"] == "host":
        return {"U": q.permute(1, 2, 3, 0).contiguous(), "dt": dts}
    got = {"state": q, "dt": np.array(dts[-c["steps"]:])}
    if c["lmax"] >= 0 and not c["fp32"]:
        got["phi"] = phi
    return got
