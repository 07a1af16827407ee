"""Edges of the analysis without an eigensolver (csrc/letkf_direct.cu) through the allocation-free
entry point: windows whose observations weigh nothing."""
import numpy as np
import pytest

from test_gpu_letkf_direct import _analyse, _case

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("sigma", [1e25, float("inf")])
@pytest.mark.parametrize("M,p,L", [(9, 1, 0), (32, 1, 0), (13, 2, 0), (32, 2, 0), (16, 4, 1), (32, 4, 1)])
def test_observations_without_weight_leave_the_inflated_ensemble(M, p, L, sigma):
    """Errors so large that every weight rounds to zero: no pattern has a table entry, and the
    analysis is xbar + sqrt(beta) dX whatever the observations hold, a NaN among them.  The
    call before it leaves the shared scratch full of another configuration's numbers.

    Bound: the mean cancels up to sqrt(beta) - 1, so that half an ulp of the population and a few
    more of rounding remain (3e-7 of the largest), and about 20 roundings of the shifted sum on
    the perturbations (4e-6 of the largest)."""
    big, F2, obs2 = _case(64, 32, 32, 1, 0, 1.1, 0.002, 1e-4)
    assert _analyse(big, F2, obs2)[1] == 0
    cfg, F, obs = _case(64, 32, M, p, L, 1.1, 0.002, 1e-4)
    cfg.obs_error_u = cfg.obs_error_rho = sigma
    obs[1][::p, ::p] = np.nan
    got, rc, st = _analyse(cfg, F, obs)
    assert rc == 0 and st[1] == 0 and st[2] == 0, (rc, st)
    F = F.astype(np.float64)
    dX = F - F.mean(0)
    want = F.mean(0) + np.sqrt(1.1) * dX
    assert np.max(np.abs(dX)) > 1e-6
    assert np.max(np.abs(got - want)) < 3e-7 * np.max(np.abs(F)) + 4e-6 * np.max(np.abs(dX))
