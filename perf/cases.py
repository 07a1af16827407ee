"""The work that users of this engine have it do, as cases with sizes, for measuring it.

A case is one pass through the public entry points of ``lbl``, as a program that runs
experiments calls them, with the sizes of the repository's workloads, tests and reference
configurations:

  forecast  update(t, n) of a whole ensemble, then the fields of the result
  analysis  lbl_letkf_analysis_noalloc on the caller's device buffers
  cycle     cycle_async per DA interval with new host observations, then the ensemble statistics
  batch     several experiments cycled together (lbl.Batch), then each one's statistics

Physics, observation errors, localisation and inflation are the DA workloads': cs 0.1, tau 0.51,
a k^4 exp(-2 (k/4)^2) initial spectrum at rms 1 (0.05 lattice units), sigma_u 0.1, sigma_rho 0.01,
inflation 1.1, an ensemble of the nature field plus 10% perturbations.  Observations are
those of a nature run, so innovations and spread are the ones a twin experiment meets.
``exact`` gives the same results in 64 bits from torch alone.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(ROOT, "lbm2d-letkf_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import lbl  # noqa: E402
from lbl.closure import load_params  # noqa: E402

PHYS = dict(cs=0.1, tau=0.51)
SIGMA_U, SIGMA_RHO, BETA, SPREAD = 0.1, 0.01, 1.1, 0.1
KF, FKF, FRICTION, H_REF, CFL = 4.0, 5.6, 5e-4, 2 * math.pi, 0.05
C_SPEED = 1.0 / CFL
BATCH = ((128, 4), (128, 8), (256, 16), (512, 32))  # the mixed batch's (grid, members)


# ---- the cases ------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one output slot (5 steps) of a single run on the reference's smallest grid
        dict(name="forecast_64_m1", kind="forecast", nx=64, ny=64, m=1, steps=5, storage="f32"),
        # a nature run between two outputs at the default cadence (iiter 20 x ioprune 10 = 200 steps)
        dict(name="forecast_256_m1", kind="forecast", nx=256, ny=256, m=1, steps=200, storage="f32"),
        # a grid that is not square and fits no specialised width, an odd ensemble and step count
        dict(name="forecast_160x104_m5", kind="forecast", nx=160, ny=104, m=5, steps=37, storage="f32"),
        # the 256^2 x 16 ensemble's free forecast over one output interval
        dict(name="forecast_256_m16", kind="forecast", nx=256, ny=256, m=16, steps=200, storage="f32"),
        # the precision form: FP16 deviations at 512^2, populations from HBM
        dict(name="forecast_512_m32_f16", kind="forecast", nx=512, ny=512, m=32, steps=100, storage="f16"),
        # one analysis at the reference's published mesh with its default window (every point observed)
        dict(name="analysis_128_m4_p1", kind="analysis", nx=128, ny=128, m=4, p=1, loc=0),
        # one analysis of the 256^2 x 16 workload (observations every 4 points, localised window)
        dict(name="analysis_256_m16_p4", kind="analysis", nx=256, ny=256, m=16, p=4, loc=1),
        # a ragged one: not square, 23 members, observations every 2 points
        dict(name="analysis_160x96_m23_p2", kind="analysis", nx=160, ny=96, m=23, p=2, loc=0),
        # two DA cycles between outputs of the 256^2 x 16 twin experiment, the headline workload
        dict(name="cycle_256_m16", kind="cycle", nx=256, ny=256, m=16, p=4, loc=1, steps=100, cycles=2,
             storage="f32", closure=0),
        # the same with the learned closure, its network every 20 steps
        dict(name="cycle_256_m16_closure", kind="cycle", nx=256, ny=256, m=16, p=4, loc=1, steps=100, cycles=2,
             storage="f32", closure=20),
        # one DA cycle of the 512^2 x 64 workload, the largest single experiment with a wide ensemble
        dict(name="cycle_512_m64", kind="cycle", nx=512, ny=512, m=64, p=4, loc=1, steps=100, cycles=1,
             storage="f32", closure=0),
        # experiments of uneven size cycled as one batch
        dict(name="batch_mixed", kind="batch", scale=1, steps=100),
    ]


def _cells(case):
    return case["nx"] * case["ny"] * case["m"]


def draw(rng):
    """A case of the listed ones' ranges: forecasts and cycles from 64 to 512 columns and 1 to 64
    members, analyses through the buffer entry point up to 32 members, small batches."""
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(("forecast", "forecast", "analysis", "analysis", "cycle", "cycle", "batch"))
    if kind == "batch":
        return dict(kind="batch", scale=rng.choice((2, 3, 4)), steps=log_int(10, 100))
    nx = 32 * log_int(2, 16)
    if kind == "forecast":
        ny = nx if rng.random() < 0.4 else max(24, min(512, int(nx * rng.uniform(0.5, 1.5))))
        m = log_int(1, 64)
        steps = log_int(5, 200)
        while nx * ny * m * steps > 512 * 512 * 64 * 100:
            m = max(1, m // 2)
        return dict(kind="forecast", nx=nx, ny=ny, m=m, steps=steps, storage=rng.choice(("f32", "f32", "f16")))
    p, loc = rng.choice(((1, 0), (2, 0), (2, 1), (4, 0), (4, 1), (8, 1)))
    ny = nx if rng.random() < 0.4 else max(4, log_int(8, 64)) * 8
    if kind == "analysis":
        m = log_int(2, 32)
        while 3 * (nx // p) * (ny // p) * (m + 1) * 4 > 7 << 20:  # the entry point's 8 MiB of scratch
            nx, ny = max(64, (nx // 64) * 32), max(32, (ny // 16) * 8)
        return dict(kind="analysis", nx=nx, ny=ny, m=m, p=p, loc=loc)
    m = log_int(4, 64)
    while nx * ny * m > 512 * 512 * 32:
        m = max(4, m // 2)
    return dict(kind="cycle", nx=nx, ny=ny, m=m, p=p, loc=loc, steps=log_int(20, 100), cycles=rng.choice((1, 2)),
                storage=rng.choice(("f32", "f32", "f16")), closure=0)


# ---- inputs -----------------------------------------------------------------------------
def _dev():
    return torch.device("cuda:0")


def _velocity(nx, ny, count, gen):
    """`count` random-phase velocity fields with E(k) ~ k^4 exp(-2 (k/4)^2) at rms 1: [count, 2, ny, nx], FP64."""
    dev = _dev()
    ky = torch.fft.fftfreq(ny, 1.0 / ny, dtype=torch.float64, device=dev)[:, None]
    kx = torch.fft.fftfreq(nx, 1.0 / nx, dtype=torch.float64, device=dev)[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    amp = torch.where(k > 0, torch.sqrt(k) * torch.exp(-(k / 4.0) ** 2), torch.zeros_like(k))
    out = torch.empty((count, 2, ny, nx), dtype=torch.float64, device=dev)
    for i in range(count):
        seed = int(torch.randint(1 << 62, (1,), generator=gen))
        g = torch.Generator(device=dev).manual_seed(seed)
        psi = torch.polar(amp, 2 * math.pi * torch.rand((ny, nx), generator=g, dtype=torch.float64, device=dev))
        u = torch.fft.ifft2(1j * ky * psi).real
        v = torch.fft.ifft2(-1j * kx * psi).real
        s = torch.rsqrt((u * u + v * v).mean())
        out[i, 0], out[i, 1] = u * s, v * s
    return out


_EX = [(q % 3) - 1 for q in range(9)]
_EY = [(q // 3) - 1 for q in range(9)]
_W = [4 / 9 if x * x + y * y == 0 else 1 / 9 if x * x + y * y == 1 else 1 / 36 for x, y in zip(_EX, _EY)]


def _feq(u, v):
    """Equilibrium populations at density 1: [..., 9, ny, nx]."""
    uu = (u * u + v * v) / C_SPEED ** 2
    f = []
    for q in range(9):
        uc = (_EX[q] * u + _EY[q] * v) / C_SPEED
        f.append(_W[q] * (1 + 3 * uc + 4.5 * uc * uc - 1.5 * uu))
    return torch.stack(f, dim=-3)


def _ensemble_f(nx, ny, m, seed, spread=SPREAD):
    """(populations of the nature run [9, ny, nx], of the members [m, 9, ny, nx]), FP32 on the GPU."""
    gen = torch.Generator().manual_seed(seed)
    nature = _velocity(nx, ny, 1, gen)[0]
    f = torch.empty((m, 9, ny, nx), dtype=torch.float32, device=_dev())
    for i in range(m):
        w = nature + (spread * _velocity(nx, ny, 1, gen)[0] if spread else 0.0)
        f[i] = _feq(w[0], w[1]).float()
    return _feq(nature[0], nature[1]).float(), f


# ---- the model in 64 bits (torch only): the truth runs and the exact results ----------------
class _Curand:
    """The forcing's normals: cuRAND's MTGP32 stream (seed 1991) in blocks of 4096 x modes, as data.cu:239-297."""

    def __init__(self, n_modes):
        self.lib = ctypes.CDLL("libcurand.so.10")
        self.g = ctypes.c_void_p()
        assert self.lib.curandCreateGenerator(ctypes.byref(self.g), 141) == 0  # CURAND_RNG_PSEUDO_MTGP32
        self.lib.curandSetPseudoRandomGeneratorSeed(self.g, ctypes.c_ulonglong(1991))
        self.n4, self.size = 4 * n_modes, 4096 * n_modes
        self.buf = torch.empty(self.size, dtype=torch.float32, device=_dev())
        self.at = self.size
        self.next()
        self.next()  # two calls at initialisation

    def next(self):
        self.at += self.n4
        if self.at + self.n4 >= self.size:
            torch.cuda.synchronize()
            assert self.lib.curandGenerateNormal(self.g, ctypes.c_void_p(self.buf.data_ptr()),
                                                 ctypes.c_size_t(self.size), ctypes.c_float(0.0),
                                                 ctypes.c_float(0.84089641525)) == 0
            torch.cuda.synchronize()
            self.at = 0
        return self.buf[self.at:self.at + self.n4].double()

    def close(self):
        self.lib.curandDestroyGenerator(self.g)


class _Model:
    """LBM steps in FP64 over f [m, 9, ny, nx]: pull streaming, Smagorinsky, BGK and the random forcing
    (lbm.cu:20-160, data.cu:161-350)."""

    def __init__(self, nx, ny):
        self.nx, self.ny = nx, ny
        self.dx = H_REF / (ny - 1)
        self.dt = self.dx / C_SPEED
        self.nu = (PHYS["tau"] - 0.5) * C_SPEED ** 2 * self.dt / 3
        k = [(x, y) for y in range(int(KF + 2)) for x in range(int(KF + 2))
             if (x or y) and KF - 2 <= math.hypot(x, y) <= KF + 2]
        a = [math.exp(-(math.hypot(x, y) - KF) ** 2) for x, y in k]
        dev = _dev()
        self.kx = torch.tensor([float(x) for x, _ in k], dtype=torch.float64, device=dev)
        self.ky = torch.tensor([float(y) for _, y in k], dtype=torch.float64, device=dev)
        amp = torch.tensor(a, dtype=torch.float64, device=dev) * (FKF / sum(a))
        X = (torch.arange(nx, dtype=torch.float64, device=dev) - nx // 2) / nx
        Y = (torch.arange(ny, dtype=torch.float64, device=dev) - ny // 2) / ny
        th = 2 * math.pi * (self.kx[:, None, None] * X[None, None, :] + self.ky[:, None, None] * Y[None, :, None])
        self.sin, self.cos = torch.sin(th), torch.cos(th)
        self.ax, self.ay = amp * 2 * math.pi * self.ky, -amp * 2 * math.pi * self.kx
        self.rand = _Curand(len(k))

    def force(self):
        n = len(self.kx)
        r = self.rand.next()
        a, b = r[:n] * self.kx + r[n:2 * n] * self.ky, r[2 * n:3 * n] * self.kx + r[3 * n:] * self.ky
        return (torch.tensordot(self.ax * a, self.sin, 1) + torch.tensordot(self.ax * b, self.cos, 1),
                torch.tensordot(self.ay * a, self.sin, 1) + torch.tensordot(self.ay * b, self.cos, 1))

    def step(self, f, force):
        """(f after one step, rho, u, v of its streaming)."""
        g = torch.stack([torch.roll(f[:, q], (_EY[q], _EX[q]), (-2, -1)) for q in range(9)], 1)
        rho, u, v = _moments(g)
        s = 1 / (2 * self.dx)
        ux, vx = ((torch.roll(a, -1, -1) - torch.roll(a, 1, -1)) * s for a in (u, v))
        uy, vy = ((torch.roll(a, -1, -2) - torch.roll(a, 1, -2)) * s for a in (u, v))
        ss = ux * ux + vy * vy + 0.5 * (uy + vx) ** 2
        nu = self.nu + (PHYS["cs"] * self.dx) ** 2 * torch.sqrt(2 * ss)
        om = 1 / (0.5 + 3 * nu / C_SPEED ** 2 / self.dt)
        uu = (u * u + v * v) / C_SPEED ** 2
        gx = (force[0] - FRICTION / self.dt * u) * self.dt
        gy = (force[1] - FRICTION / self.dt * v) * self.dt
        for q in range(9):
            uc = (_EX[q] * u + _EY[q] * v) / C_SPEED
            rw = rho * _W[q]
            g[:, q] += -om * (g[:, q] - rw * (1 + 3 * uc + 4.5 * uc * uc - 1.5 * uu)) \
                + rw * (gx * _EX[q] + gy * _EY[q]) * (3 / C_SPEED ** 2)
        return g, rho, u, v

    def run(self, f, n):
        """n steps; members in groups, so that the temporaries stay small."""
        per = max(1, (1 << 22) // (self.nx * self.ny))
        forces = [self.force() for _ in range(n)]
        mac = torch.empty((f.shape[0], 3, self.ny, self.nx), dtype=torch.float64, device=f.device)
        for a in range(0, f.shape[0], per):
            h = f[a:a + per]
            for k in range(n):
                h, r, u, v = self.step(h, forces[k])
            f[a:a + per] = h
            mac[a:a + per, 0], mac[a:a + per, 1], mac[a:a + per, 2] = r, u, v
        return f, mac

    def vorticity(self, u, v):
        s = 1 / (2 * self.dx)
        return (torch.roll(v, -1, -1) - torch.roll(v, 1, -1)) * s - (torch.roll(u, -1, -2) - torch.roll(u, 1, -2)) * s

    def stats(self, mac):
        w = self.vorticity(mac[:, 1], mac[:, 2])
        return tuple(a.cpu().numpy() for a in (mac[:, 1].mean(0), mac[:, 2].mean(0), w.mean(0), w.std(0, correction=0)))


def _moments(f):
    rho = f.sum(1)
    u = sum(_EX[q] * f[:, q] for q in range(9) if _EX[q]) * C_SPEED / rho
    v = sum(_EY[q] * f[:, q] for q in range(9) if _EY[q]) * C_SPEED / rho
    return rho, u, v


def _gaspari_cohn(d):
    if d <= 0:
        return 1.0
    if d <= 1:
        return -d ** 5 / 4 + d ** 4 / 2 + d ** 3 * 5 / 8 - d * d * 5 / 3 + 1
    if d <= 2:
        return d ** 5 / 12 - d ** 4 / 2 + d ** 3 * 5 / 8 + d * d * 5 / 3 - 5 * d + 4 - 2 / 3 / d
    return 0.0


def _inverse_sqrt(Q):
    """Q^-1/2 of a batch of symmetric positive definite matrices: the coupled Newton-Schulz iteration."""
    s = torch.linalg.matrix_norm(Q, float("inf"))[:, None, None]
    eye = torch.eye(Q.shape[-1], dtype=Q.dtype, device=Q.device)
    Y, Z = Q / s, eye.expand_as(Q).clone()
    for _ in range(60):
        T = 1.5 * eye - 0.5 * (Z @ Y)
        Y, Z = Y @ T, T @ Z
        if float((T - eye).abs().max()) < 1e-13:
            break
    return Z / torch.sqrt(s)


def _analyse(f, yo, p, loc):
    """The LETKF analysis of f [m, 9, ny, nx] (FP64) with the site observations yo [3, ny/p, nx/p] (u, v, rho),
    and the moments of the analysis (letkf.cu:29-360, letkf_solver.h:235-349)."""
    m, _, ny, nx = f.shape
    if loc <= 0:
        dloc, nl, off, nox = p - 1, 0 if p == 1 else 2, 0 if p == 1 else 1, 1 if p == 1 else 4
    else:
        dloc, nl, off, nox = loc * p, 2 * loc, 0, 4 * loc + 1
    rho, u, v = _moments(f[:, :, ::p, ::p])
    H = torch.stack([u, v, rho], 0)                                   # [3, m, nsy, nsx]
    dY, dyo = H - H.mean(1, keepdim=True), yo - H.mean(1)
    sig2 = (SIGMA_U ** 2, SIGMA_U ** 2, SIGMA_RHO ** 2)
    out = torch.empty_like(f)
    for pj in range(p):
        for pi in range(p):
            rows, inno = [], []
            for b in range(nox):
                for a in range(nox):
                    da, db = a - (nl - off), b - (nl - off)
                    di, dj = pi - da * p, pj - db * p
                    if max(abs(di), abs(dj)) > nl * p:
                        continue
                    w = _gaspari_cohn(math.hypot(di, dj) / (dloc + 1e-6)) if p > 1 else 1.0
                    if not w > 0:
                        continue
                    for var in range(3):
                        sw = math.sqrt(w / sig2[var])
                        rows.append(sw * torch.roll(dY[var], (-db, -da), (-2, -1)))
                        inno.append(sw * torch.roll(dyo[var], (-db, -da), (-2, -1)))
            C = torch.stack(rows, 0).flatten(2).permute(2, 0, 1)      # [points, obs, m]
            d = torch.stack(inno, 0).flatten(1).T                     # [points, obs]
            X = f[:, :, pj::p, pi::p].flatten(2).permute(2, 1, 0)     # [points, 9, m]
            A = torch.empty_like(X)
            step = max(1, (1 << 24) // (m * m))
            for k in range(0, X.shape[0], step):
                c, x = C[k:k + step], X[k:k + step]
                Q = (m - 1) / BETA * torch.eye(m, dtype=f.dtype, device=f.device) + c.transpose(1, 2) @ c
                Z = _inverse_sqrt(Q)
                wa = Z @ (Z @ (c.transpose(1, 2) @ d[k:k + step, :, None]))
                xb = x.mean(2, keepdim=True)
                A[k:k + step] = xb + (x - xb) @ (math.sqrt(m - 1) * Z + wa)
            out[:, :, pj::p, pi::p] = A.permute(2, 1, 0).reshape(m, 9, ny // p, nx // p)
    return out, _moments(out)


def _truth(nx, ny, f_nature, cycles, steps, seed):
    """Noisy (rho, u, v) fields of a nature run at the end of each DA interval: the observations, NaN-free off
    the lattice as the engine never reads there."""
    model = _Model(nx, ny)
    f = f_nature.double()[None]
    gen = torch.Generator(device=_dev()).manual_seed(seed + 17)
    obs = []
    for _ in range(cycles):
        f, mac = model.run(f, steps)
        noise = torch.randn(mac[0].shape, generator=gen, dtype=torch.float64, device=_dev())
        noise *= torch.tensor([SIGMA_RHO, SIGMA_U, SIGMA_U], dtype=torch.float64, device=_dev())[:, None, None]
        obs.append(tuple(np.ascontiguousarray(a) for a in (mac[0] + noise).float().cpu().numpy()))
    model.rand.close()
    return obs


# ---- states ----------------------------------------------------------------------------
def _config(mode, nx, ny, m, **kw):
    return lbl.config_default(mode, nx, m, ny=ny, ic_kind=lbl.IC_K4EXP, ic_amp=1.0, **PHYS, **kw)


def _ensemble(cfg, f, closure=0):
    ens = lbl.Ensemble(cfg)
    if closure:
        params, meta = load_params()
        ens.set_closure(params, meta["nu_ref"], meta["dx_ref"])
        ens.set_closure_refresh(closure)
    ens.init(0)
    for i in range(f.shape[0]):
        ens.set_f(i, f[i].cpu().numpy())
    return ens


def _da_config(nx, ny, m, p, loc, steps, storage="f32"):
    return _config("DA_LETKF", nx, ny, m, da_xyprune=p, letkf_rloc_len=loc, letkf_covinf=BETA, obs_error_u=SIGMA_U,
                   obs_error_rho=SIGMA_RHO, iiter=steps, daprune=1,
                   storage=lbl.STORAGE_F16 if storage == "f16" else lbl.STORAGE_F32)


OBS_CYCLES = 4  # DA intervals of the nature run that a state's observations cover, then taken again


def _experiment(nx, ny, m, p, loc, steps, seed, storage="f32", closure=0):
    nature, f = _ensemble_f(nx, ny, m, seed)
    ens = _ensemble(_da_config(nx, ny, m, p, loc, steps, storage), f, closure)
    return ens, _truth(nx, ny, nature, OBS_CYCLES, steps, seed)


def _analysis_inputs(case, seed):
    nx, ny, m, p = case["nx"], case["ny"], case["m"], case["p"]
    nature, f = _ensemble_f(nx, ny, m, seed)
    rho, u, v = _moments(nature[None, :, ::p, ::p].double())
    gen = torch.Generator(device=_dev()).manual_seed(seed + 29)
    yo = torch.stack([u[0], v[0], rho[0]])
    noise = torch.randn(yo.shape, generator=gen, dtype=torch.float64, device=_dev())
    yo = yo + noise * torch.tensor([SIGMA_U, SIGMA_U, SIGMA_RHO], dtype=torch.float64, device=_dev())[:, None, None]
    return f, yo.float().contiguous()


def _batch_sizes(case):
    return [(max(128, nx // case["scale"] // 128 * 128), max(2, m // case["scale"])) for nx, m in BATCH]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "forecast":
        f = _ensemble_f(case["nx"], case["ny"], case["m"], seed, SPREAD if case["m"] > 1 else 0.0)[1]
        cfg = _config("NATURE", case["nx"], case["ny"], case["m"],
                      storage=lbl.STORAGE_F16 if case["storage"] == "f16" else lbl.STORAGE_F32)
        return dict(case=case, ens=_ensemble(cfg, f), t=0)
    if kind == "analysis":
        f, yo = _analysis_inputs(case, seed)
        cfg = _da_config(case["nx"], case["ny"], case["m"], case["p"], case["loc"], 20)
        mac = torch.zeros((case["m"], 3, case["ny"], case["nx"]), dtype=torch.float32, device=_dev())
        return dict(case=case, cfg=cfg, f=f, yo=yo, out=torch.empty_like(f), mac=mac, lib=lbl.load_library())
    if kind == "cycle":
        ens, obs = _experiment(case["nx"], case["ny"], case["m"], case["p"], case["loc"], case["steps"], seed,
                               case["storage"], case["closure"])
        return dict(case=case, ens=ens, obs=obs, k=0, t=0)
    exps = [_experiment(nx, nx, m, 4, 1, case["steps"], seed + 101 * i)
            for i, (nx, m) in enumerate(_batch_sizes(case))]
    return dict(case=case, batch=lbl.Batch([e for e, _ in exps]), exps=[e for e, _ in exps],
                obs=[o for _, o in exps], k=0, t=0)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forecast":
        ens, n = state["ens"], case["steps"]
        ens.update(state["t"], n)
        state["t"] += n
        return ens.get_fields(0) if case["m"] == 1 else ens.ens_stats()
    if kind == "analysis":
        rc = state["lib"].lbl_letkf_analysis_noalloc(
            ctypes.byref(state["cfg"]), state["f"].data_ptr(), state["out"].data_ptr(), state["mac"].data_ptr(),
            state["yo"].data_ptr(), torch.cuda.current_stream().cuda_stream, None, None, 0)
        if rc != 0:
            raise lbl.LblError(rc, "lbl_letkf_analysis_noalloc")
        return state["out"], state["mac"]
    if kind == "cycle":
        ens, n = state["ens"], case["steps"]
        for _ in range(case["cycles"]):
            state["t"] += n
            ens.cycle_async(state["t"], *state["obs"][state["k"] % OBS_CYCLES], n)
            state["k"] += 1
        return ens.ens_stats()
    state["t"] += case["steps"]
    state["batch"].cycle_async(state["t"], [o[state["k"] % OBS_CYCLES] for o in state["obs"]], case["steps"])
    state["k"] += 1
    state["batch"].sync()
    return [e.ens_stats() for e in state["exps"]]


# ---- work: what a pass cannot do without ---------------------------------------------------
LBM_FLOPS = 170.0  # per cell and step: moments, strain, relaxation, nine directions' collision and force


def _analysis_work(nx, ny, m, p, loc):
    """Site ensembles and populations in, analysis and moments out; the local matrices' products and one
    tridiagonal reduction of the smaller of the member and observation spaces."""
    obs = 3 * (1 if p == 1 and loc <= 0 else max(1.0, math.pi * (2.0 * (max(1, loc) * p if loc else p - 1) / p) ** 2))
    n = min(m, obs)
    flops = 2 * obs * m * n + 4 / 3 * n ** 3 + 4 * 9 * m * n
    return dict(bytes=4.0 * nx * ny * m * (9 + 9 + 2) + 12.0 * (nx // p) * (ny // p), flops=flops * nx * ny)


def _forecast_work(nx, ny, m, steps, elem):
    return dict(bytes=nx * ny * (m * (9 * elem * 2 + 12.0)), flops=LBM_FLOPS * nx * ny * m * steps)


def _add(a, b):
    return dict(bytes=a["bytes"] + b["bytes"], flops=a["flops"] + b["flops"])


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = dict(bytes=0.0, flops=0.0)
        for nx, m in _batch_sizes(case):
            total = _add(total, _add(_forecast_work(nx, nx, m, case["steps"], 4), _analysis_work(nx, nx, m, 4, 1)))
        return total
    nx, ny, m = case["nx"], case["ny"], case["m"]
    if kind == "analysis":
        return _analysis_work(nx, ny, m, case["p"], case["loc"])
    elem = 2 if case["storage"] == "f16" else 4
    if kind == "forecast":
        return _forecast_work(nx, ny, m, case["steps"], elem)
    one = _add(_forecast_work(nx, ny, m, case["steps"], elem), _analysis_work(nx, ny, m, case["p"], case["loc"]))
    return dict(bytes=one["bytes"] * case["cycles"], flops=one["flops"] * case["cycles"])


# ---- exact results ---------------------------------------------------------------------
def _exact_cycles(nx, ny, m, p, loc, steps, cycles, seed):
    nature, f = _ensemble_f(nx, ny, m, seed)
    obs = _truth(nx, ny, nature, cycles, steps, seed)
    model = _Model(nx, ny)
    f = f.double()
    for k in range(cycles):
        ro, uo, vo = (torch.from_numpy(a).to(_dev()).double()[::p, ::p] for a in obs[k])
        f, _ = _analyse(f, torch.stack([uo, vo, ro]), p, loc)
        f, mac = model.run(f, steps)
    model.rand.close()
    return model.stats(mac)


def exact(case, seed):
    """What the first pass on prepare(case, seed) returns, in 64 bits; None with the learned closure, whose
    network is defined in 16 bits."""
    kind = case["kind"]
    if kind == "forecast":
        f = _ensemble_f(case["nx"], case["ny"], case["m"], seed, SPREAD if case["m"] > 1 else 0.0)[1].double()
        model = _Model(case["nx"], case["ny"])
        f, mac = model.run(f, case["steps"])
        model.rand.close()
        if case["m"] > 1:
            return model.stats(mac)
        w = model.vorticity(mac[0, 1], mac[0, 2])
        return tuple(a.cpu().numpy() for a in (mac[0, 0], mac[0, 1], mac[0, 2], w))
    if kind == "analysis":
        f, yo = _analysis_inputs(case, seed)
        a, (rho, u, _) = _analyse(f.double(), yo.double(), case["p"], case["loc"])
        return a, torch.stack([rho, u, torch.zeros_like(u)], 1)
    if kind == "cycle":
        if case["closure"]:
            return None
        return _exact_cycles(case["nx"], case["ny"], case["m"], case["p"], case["loc"], case["steps"], case["cycles"],
                             seed)
    return [_exact_cycles(nx, nx, m, 4, 1, case["steps"], 1, seed + 101 * i)
            for i, (nx, m) in enumerate(_batch_sizes(case))]
