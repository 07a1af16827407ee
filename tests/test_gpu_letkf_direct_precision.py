"""Errors against FP64 of the analyses without an eigensolver (csrc/letkf_direct.cu) and of the
Jacobi kernels, on inputs whose FP32 observation operator is exact: what is compared is the
solvers alone.  The perturbations are multiples of 2^-16 that sum to zero over the members and
leave the density at exactly 1, so that every sum, mean and quotient of the operator is exact;
the rest population holds what the others leave and is not compared."""
import numpy as np
import pytest

import lbl
from test_gpu_letkf_direct import _analyse, _oracle
from test_gpu_letkf_direct_agreement import _assimilate

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

Q = [0, 1, 2, 3, 5, 6, 7, 8]


def _exact_case(nx, ny, M, p, L, sigma, seed=3):
    """(configuration, populations, observations (rho, u, v)): perturbations of rms 2^-6, smooth
    over 8 wavenumbers, observed with the error sigma."""
    rng = np.random.default_rng(seed)
    k2 = np.fft.fftfreq(ny, 1 / ny)[:, None] ** 2 + np.fft.rfftfreq(nx, 1 / nx)[None] ** 2
    a = np.fft.irfft2(np.fft.rfft2(rng.standard_normal((M, 9, ny, nx))) * np.exp(-k2 / 64.0), s=(ny, nx))
    step = 2.0 ** -16
    f = np.round(a / a.std() * 2.0 ** -6 / step) * step
    f[-1] = -f[:-1].sum(0)
    f[:, 4] = 0
    f[:, 4] = 1 - f.sum(1)
    o = 2.0 ** -12
    u, v = np.round(0.3 * rng.standard_normal((2, ny, nx)) / o) * o
    rho = 1 + np.round(1e-2 * rng.standard_normal((ny, nx)) / o) * o
    cfg = lbl.config_default("DA_LETKF", nx, M, ny=ny, da_xyprune=p, letkf_rloc_len=L, letkf_covinf=1.1,
                             obs_error_u=sigma, obs_error_rho=sigma, daprune=1)
    F = f.astype(np.float32)
    assert np.array_equal(F, f)
    return cfg, F, [x.astype(np.float32) for x in (rho, u, v)]


def _errors(cfg, F, obs):
    """rms error, in units of the largest increment, of (the entry point, lbl_assimilate), and the
    largest condition number."""
    got, rc, st = _analyse(cfg, F, obs)
    assert rc == 0 and st[2] == 0, (rc, st)
    jac = _assimilate(cfg, F, obs)
    want, lam = _oracle(cfg, F, obs)
    scale = np.max(np.abs(want - F)[:, Q])
    rms = [float(np.sqrt(np.mean((x - want)[:, Q] ** 2)) / scale) for x in (got, jac)]
    kappa = float(np.max(lam.max(-1) / lam.min(-1)))
    print(f"M={cfg.n_ens} p={cfg.da_xyprune} L={cfg.letkf_rloc_len} kappa {kappa:.1e}: {rms[0]:.2e}, Jacobi {rms[1]:.2e}")
    return rms[0], rms[1], kappa


@pytest.mark.parametrize("M,p,L,sigma", [
    (16, 1, 1, 1.0), (16, 1, 1, 0.3), (9, 1, 1, 0.1), (12, 2, 1, 0.1), (16, 4, 1, 0.1), (16, 2, 2, 0.1),
    (32, 1, 1, 0.3), (24, 4, 1, 0.03), (32, 4, 0, 0.1), (32, 2, 2, 0.1),
])
def test_primal_error_is_no_larger_than_the_jacobi_kernels(M, p, L, sigma):
    """The Gram's roundings decide the error from kappa 1e3 on.  Bound: the Jacobi kernel's error on
    the same inputs, with a tenth for the draw."""
    got, jac, _ = _errors(*_exact_case(64, 32, M, p, L, sigma))
    assert got < 1.1 * jac


@pytest.mark.parametrize("sigma", [3e-2, 1e-2, 1e-3, 3e-4, 1e-4])
@pytest.mark.parametrize("M,p,L", [(16, 1, 1), (32, 1, 1), (24, 4, 1)])
def test_ill_conditioned_points_are_the_jacobi_kernels(M, p, L, sigma):
    """Condition numbers from 1e4 (a part of the tiles) to 1e9, where the reduction would lose to the
    iteration.  A tile above the limit has lbl_assimilate's very populations; up to kappa 1e8,
    where they are still an analysis, none is further from FP64 than they are (a tenth for the
    draw); beyond, the points that did not converge are counted."""
    cfg, F, obs = _exact_case(64, 32, M, p, L, sigma)
    got, rc, st = _analyse(cfg, F, obs)
    jac = _assimilate(cfg, F, obs)
    want, lam = _oracle(cfg, F, obs)
    assert rc == 0 and np.isfinite(got).all() and st[3] >= 64 * 32
    same = (got == jac).all((0, 1))
    kappa = lam.max(-1) / lam.min(-1)
    print(f"kappa {kappa.max():.1e}, {same.mean():.3f} of the points by the iteration, counters {st}")
    assert same[kappa > 4e4].all()
    if kappa.max() < 2e8:
        rms = [np.sqrt(np.mean((x - want)[:, Q] ** 2)) for x in (got, jac)]
        assert st[1] == 0 and rms[0] < 1.1 * rms[1]
    if kappa.max() > 5e8:
        assert st[1] > 0


@pytest.mark.parametrize("M", [16, 32])
@pytest.mark.parametrize("sigma", [1e-1, 1e-2, 1e-3, 1e-4])
def test_dual_error_is_no_larger_than_the_jacobi_kernels(M, sigma):
    """Fifteen observations (order 16), kappa 1e3 to 1e9: at most the Jacobi kernel's error, and the
    points of the last are counted as not converged, as the iteration counts them."""
    cfg, F, obs = _exact_case(64, 32, M, 2, 0, sigma)
    got, jac, kappa = _errors(cfg, F, obs)
    assert got < jac
    assert (_analyse(cfg, F, obs)[2][1] > 0) == (kappa > 1e8)


@pytest.mark.parametrize("k", range(19))
def test_pointwise_error_over_every_table_of_shifts(k):
    """Three observations (order 8) at errors of 2^-k: each step multiplies kappa by 4, from 4^2 to 4^20,
    so that every table of shifts is met.  FP64 from the singular values of the 3 x M matrix.

    Bound: rms 1e-7 of the largest increment: half an ulp of a population and one of the
    perturbation, 2^-24 each, and as much for the sums."""
    M, sigma, beta = 16, 2.0 ** -k, 1.1
    cfg, F, obs = _exact_case(32, 16, M, 1, 0, sigma)
    got, rc, st = _analyse(cfg, F, obs)
    assert rc == 0 and st[:3] == [1, 0, 0]
    f = F.astype(np.float64)
    ex, ey = np.arange(9) % 3 - 1, np.arange(9) // 3 - 1
    c = cfg.u_ref / cfg.cfl
    rho = f.sum(1)
    H = np.stack([(f * ex[:, None, None]).sum(1) * c / rho, (f * ey[:, None, None]).sum(1) * c / rho, rho])
    yo = np.stack([obs[1], obs[2], obs[0]]).astype(np.float64)
    C = ((H - H.mean(1, keepdims=True)) / sigma).transpose(2, 3, 0, 1)
    d = ((yo - H.mean(1)) / sigma).transpose(1, 2, 0)
    U, s, Vt = np.linalg.svd(C, full_matrices=False)
    a = (M - 1) / beta
    X = f.transpose(2, 3, 1, 0)
    dX = X - X.mean(-1, keepdims=True)
    P = dX @ Vt.swapaxes(-1, -2)
    e = np.sqrt(M - 1) * (1 / np.sqrt(a + s * s) - 1 / np.sqrt(a))
    A = X.mean(-1, keepdims=True) + np.sqrt(beta) * dX + (P * e[..., None, :]) @ Vt
    A += (P * (s / (a + s * s))[..., None, :]) @ (U.swapaxes(-1, -2) @ d[..., None])
    want = A.transpose(3, 2, 0, 1)
    scale = np.max(np.abs(want - f)[:, Q])
    rms = np.sqrt(np.mean((got - want)[:, Q] ** 2)) / scale
    print(f"kappa {1 + np.max(s) ** 2 / a:.1e}: rms {rms:.2e}")
    assert rms < 1e-7
