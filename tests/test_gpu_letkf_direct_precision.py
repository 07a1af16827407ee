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
