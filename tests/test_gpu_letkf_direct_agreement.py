"""The allocation-free entry point's analyses without an eigensolver (csrc/letkf_direct.cu) against
the Jacobi kernels of lbl_assimilate on the same forecasts and observations.  Both centre the
same FP32 operator, so its error drops out and what remains is the two solvers'.

Bound: 3e-5 of the largest increment (the Jacobi iteration's share of a run's sweeps is about
2e-5), and three roundings of a population."""
import numpy as np
import pytest

import lbl
from test_gpu_letkf_direct import _analyse, _case

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _assimilate(cfg, F, obs):
    """The same analysis by lbl_assimilate, FP64 copies of its populations."""
    e = lbl.Ensemble(cfg)
    e.init(0)
    for m in range(F.shape[0]):
        e.set_f(m, F[m])
    e.assimilate(cfg.iiter, *obs)
    out = np.stack([e.get_f(m) for m in range(F.shape[0])]).astype(np.float64)
    e.close()
    return out


def _check(nx, ny, M, p, L):
    cfg, F, obs = _case(nx, ny, M, p, L, 1.1, 0.002, 1e-4)
    got, rc, st = _analyse(cfg, F, obs)
    want = _assimilate(cfg, F, obs)
    assert rc == 0 and st[1] == 0 and st[2] == 0, (rc, st)
    scale, top = np.max(np.abs(want - F)), np.max(np.abs(F))
    err = np.max(np.abs(got - want))
    print(f"{nx}x{ny} M={M} p={p} L={L}: {err / scale:.2e} of the largest increment {scale:.2e}")
    assert scale > 1e-6 and err < 3e-5 * scale + 3 * 2.0 ** -24 * top


@pytest.mark.parametrize("M", [9, 16, 17, 32])
@pytest.mark.parametrize("nx,ny", [(64, 32), (96, 20)])
def test_pointwise_windows(nx, ny, M):
    """Three observations a point, order 8 on sixteen lanes: eight lanes hold no matrix row, and
    their zeros must not reach the reflections."""
    _check(nx, ny, M, 1, 0)


@pytest.mark.parametrize("M,p,L", [(9, 1, 0), (16, 4, 1), (32, 2, 0), (32, 4, 1)])
def test_the_iterations_options_choose_it(M, p, L):
    """A tolerance or a sweep limit of the caller's own is the Jacobi iteration's: it solves every
    point, with lbl_assimilate's bits under the same options, and the counters are its own."""
    cfg, F, obs = _case(64, 32, M, p, L, 1.1, 0.002, 1e-4)
    cfg.jacobi_tol = 1e-4
    got, rc, st = _analyse(cfg, F, obs)
    assert rc == 0 and st[0] > 1 and st[3] > 64 * 32
    np.testing.assert_array_equal(got, _assimilate(cfg, F, obs))
    cfg.jacobi_tol, cfg.jacobi_max_sweeps = 1e-6, 1
    got, rc, st = _analyse(cfg, F, obs)
    assert rc == 0 and st[0] == 1 and st[1] > 0 and st[3] == 64 * 32
    np.testing.assert_array_equal(got, _assimilate(cfg, F, obs))


@pytest.mark.parametrize("nx,ny,M,p,L", [
    (64, 32, 9, 4, 1), (64, 32, 16, 4, 1), (64, 32, 17, 4, 1), (64, 32, 32, 4, 1), (64, 32, 16, 2, 0), (96, 36, 32, 2, 0),
])
def test_every_form(nx, ny, M, p, L):
    """The smallest and largest ensembles of both member orders, and the observation space's order 16."""
    _check(nx, ny, M, p, L)
