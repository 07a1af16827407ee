"""The analysis without an eigensolver (csrc/letkf_direct.cu), through the allocation-free entry
point, against the FP64 oracle at the edges of its variants: the smallest and largest
ensembles of each order, windows with fewer observations than members (the dual form) and with
more, odd ensembles, observation blocks that do not fill a tile, and grids that are not
square; and the ensembles up to 8 members, which the Jacobi kernel serves.

Bound: the increments' of the analysis parity tests (test_gpu_letkf.py), 1e-3 of the
largest.  It is the observation operator's: u and v cancel O(0.1) populations in FP32, an error
of about 1e-6 against an observation error of 0.002 here."""
import ctypes

import numpy as np
import pytest

import lbl
import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _case(nx, ny, M, p, L, beta, sig_u, sig_r):
    """(configuration, forecast populations [M][9][ny][nx], observations (rho, u, v))."""
    cfg = lbl.config_default("DA_LETKF", nx, M, ny=ny, da_xyprune=p, letkf_rloc_len=L, letkf_covinf=beta,
                             obs_error_u=sig_u, obs_error_rho=sig_r, daprune=1)
    e = lbl.Ensemble(cfg)
    e.init(0)
    e.update(0, 20)
    F = np.stack([e.get_f(m) for m in range(M)])
    e.close()
    nat = lbl.Ensemble(lbl.config_default("NATURE", nx, 1, ny=ny))
    nat.init(0)
    nat.update(0, 20)
    fields = nat.get_fields(0)[:3]
    nat.close()
    rng = np.random.default_rng(M + 7 * p + 100 * L)
    obs = [(a + s * rng.standard_normal(a.shape)).astype(np.float32) for a, s in zip(fields, (sig_r, sig_u, sig_u))]
    return cfg, F, obs


def _analyse(cfg, F, obs):
    """(analysis populations, status, counters) of lbl_letkf_analysis_noalloc."""
    p = cfg.da_xyprune
    d_in = torch.from_numpy(F).cuda()
    d_out = torch.full_like(d_in, float("nan"))
    mac = torch.zeros((F.shape[0], 3) + F.shape[2:], device="cuda")
    yo = torch.from_numpy(np.stack([obs[k][::p, ::p] for k in (1, 2, 0)]).copy()).cuda()
    stats = (ctypes.c_int * 4)()
    rc = lbl.load_library().lbl_letkf_analysis_noalloc(ctypes.byref(cfg), d_in.data_ptr(), d_out.data_ptr(),
                                                       mac.data_ptr(), yo.data_ptr(),
                                                       torch.cuda.current_stream().cuda_stream, stats, None, 0)
    return d_out.cpu().numpy().astype(np.float64), rc, list(stats)


def _oracle(cfg, F, obs):
    o = oracle.Oracle(cfg)
    for m in range(F.shape[0]):
        o.set_f(m, F[m])
    _, lam = o.assimilate(*obs, want_lambda=True)
    want = np.stack([o.get_f(m) for m in range(F.shape[0])])
    o.close()
    return want, lam


@pytest.mark.parametrize("nx,ny,M,p,L", [
    # up to 8 members: the Jacobi kernel
    (32, 16, 2, 4, 1), (64, 32, 8, 1, 0),
    # primal, order M: 16, 32 unknowns and their first and last ensembles
    (64, 32, 9, 4, 1), (64, 32, 15, 4, 1), (64, 32, 16, 4, 1), (64, 32, 17, 4, 1),
    (64, 32, 31, 4, 1), (64, 32, 32, 4, 1), (64, 32, 32, 4, 0),
    # dual, order = observations: 3 (pointwise) and up to 12
    (32, 8, 9, 1, 0), (64, 24, 32, 1, 0), (64, 32, 13, 2, 0), (64, 32, 32, 2, 0),
    # blocks that leave a tile partly empty, one block for the whole grid, wide windows
    (96, 36, 12, 3, 1), (96, 36, 30, 3, 0), (32, 16, 16, 16, 0), (64, 32, 16, 4, 2), (64, 32, 20, 2, 1), (64, 32, 16, 1, 1),
])
def test_direct_analysis_matches_oracle(nx, ny, M, p, L):
    cfg, F, obs = _case(nx, ny, M, p, L, 1.1, 0.002, 1e-4)
    got, rc, st = _analyse(cfg, F, obs)
    want, _ = _oracle(cfg, F, obs)
    assert rc == 0 and st[0] >= 1 and st[1] == 0 and st[2] == 0 and st[3] >= nx * ny, st
    scale = np.max(np.abs(want - F))
    err = np.max(np.abs(got - want)) / scale
    print(f"{nx}x{ny} M={M} p={p} L={L}: {err:.2e} of the largest increment {scale:.2e}")
    assert scale > 1e-6 and err < 1e-3


@pytest.mark.parametrize("M,p,L,sig", [(16, 4, 1, 1e-5), (32, 4, 1, 1e-5), (32, 1, 0, 1e-6), (16, 4, 1, 1e3)])
def test_direct_analysis_over_condition_numbers(M, p, L, sig):
    """Observation errors far below and above the spread: condition numbers of Q from 1 to about 1e7,
    that is every length of the shifted sum.  At a condition number kappa the FP32 matrix itself moves
    the increments by about 6e-8 kappa; the bound is that, with a factor of 10, and at least 1e-3."""
    cfg, F, obs = _case(64, 32, M, p, L, 1.1, sig, sig)
    got, rc, st = _analyse(cfg, F, obs)
    want, lam = _oracle(cfg, F, obs)
    kappa = float(np.max(lam) / np.min(lam))
    scale = max(np.max(np.abs(want - F)), 1e-4)
    err = np.max(np.abs(got - want)) / scale
    print(f"M={M} p={p} sigma={sig}: kappa {kappa:.1e}, {err:.2e} of the largest increment")
    assert rc == 0 and err < max(1e-3, 10 * 6e-8 * kappa)


def test_direct_analysis_reports_a_nan_only_where_it_is_observed():
    """A NaN observation reaches exactly the points whose window holds its site."""
    cfg, F, obs = _case(64, 32, 16, 4, 1, 1.1, 0.002, 1e-4)
    obs[1][0, 0] = np.nan
    got, rc, st = _analyse(cfg, F, obs)
    assert rc == -5 and st[2] == 1
    bad = np.isnan(got[5]).any(0)
    dj = np.minimum(np.arange(32), 32 - np.arange(32))[:, None]
    di = np.minimum(np.arange(64), 64 - np.arange(64))[None, :]
    d = np.hypot(dj, di)
    assert bad[d < 7.9].all() and not bad[d > 8.0].any()  # twice the localisation length of 4 cells
