"""Edges of the analysis without an eigensolver (csrc/letkf_direct.cu) through the allocation-free
entry point: windows whose observations weigh nothing, tiles left to the Jacobi kernel, and blocks that several CTAs share."""
import ctypes
import time

import numpy as np
import pytest

import lbl
from test_gpu_letkf_direct import _analyse, _case
from test_gpu_letkf_direct_agreement import _assimilate
from test_gpu_letkf_direct_precision import _exact_case

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


def _call(cfg, d_in, d_out, d_mac, d_yo):
    stats = (ctypes.c_int * 4)()
    rc = lbl.load_library().lbl_letkf_analysis_noalloc(ctypes.byref(cfg), d_in.data_ptr(), d_out.data_ptr(),
                                                       d_mac.data_ptr(), d_yo.data_ptr(),
                                                       torch.cuda.current_stream().cuda_stream, stats, None, 0)
    return rc, list(stats)


@pytest.mark.parametrize("M", [16, 32])
def test_points_left_to_the_iteration(M):
    """Half of the grid has a spread of a hundred times the observation error and half a
    thousandth of that: some tiles are left to the Jacobi kernel.  No mark stays in the moments, which are
    those of the populations, every point is counted, an analysis in place is the same, and so
    is a second call."""
    nx, ny, p = 96, 36, 3
    cfg, F, obs = _exact_case(nx, ny, M, p, 1, 3e-3)
    cfg.compat_stale_v = 0
    half = F[:, :, :, nx // 2:]
    F[:, :, :, nx // 2:] = half.mean(0) + np.float32(1e-3) * (half - half.mean(0))
    d_yo = torch.from_numpy(np.stack([obs[k][::p, ::p] for k in (1, 2, 0)]).copy()).cuda()
    d_in = torch.from_numpy(F).cuda()
    out = torch.full_like(d_in, float("nan"))
    mac = torch.full((M, 3, ny, nx), float("nan"), device="cuda")
    rc, st = _call(cfg, d_in, out, mac, d_yo)
    assert rc == 0 and st[1] == 0 and st[2] == 0 and st[0] > 1 and nx * ny < st[3] < st[0] * nx * ny, (rc, st)
    f = out.cpu().numpy().astype(np.float64)
    rho = f.sum(1)
    ex, ey = np.arange(9) % 3 - 1, np.arange(9) // 3 - 1
    c = cfg.u_ref / cfg.cfl
    got = mac.cpu().numpy()
    np.testing.assert_allclose(got[:, 0], rho, rtol=1e-6)  # nine roundings of terms up to 1
    np.testing.assert_allclose(got[:, 1], (f * ex[:, None, None]).sum(1) * c / rho, atol=2e-5)  # the same times c = 20
    np.testing.assert_allclose(got[:, 2], (f * ey[:, None, None]).sum(1) * c / rho, atol=2e-5)
    again, mac2 = d_in.clone(), torch.zeros_like(mac)
    assert _call(cfg, again, again, mac2, d_yo) == (0, st)
    assert torch.equal(again, out) and torch.equal(mac2, mac)


@pytest.mark.parametrize("M", [9, 32])
@pytest.mark.parametrize("nx,ny,p,L", [
    (64, 20, 4, 1), (96, 32, 8, 1), (288, 18, 9, 1), (160, 20, 10, 0), (64, 64, 16, 1), (64, 64, 64, 1),
])
def test_blocks_shared_by_several_ctas(nx, ny, M, p, L):
    """Blocks of p x p points from one round of a CTA to many: from 9 or 10 on, several CTAs share a
    block.  Every point is analysed, and counted, once."""
    cfg, F, obs = _exact_case(nx, ny, M, p, L, 0.3)
    d_yo = torch.from_numpy(np.stack([obs[k][::p, ::p] for k in (1, 2, 0)]).copy()).cuda()
    d_in = torch.from_numpy(F).cuda()
    out = torch.full_like(d_in, float("nan"))
    rc, st = _call(cfg, d_in, out, torch.zeros((M, 3, ny, nx), device="cuda"), d_yo)
    assert (rc, st) == (0, [1, 0, 0, nx * ny])
    want = _assimilate(cfg, F, obs)
    scale = np.max(np.abs(want - F))
    assert scale > 1e-4 and np.max(np.abs(out.cpu().numpy() - want)) < 3e-5 * scale + 3 * 2.0 ** -24


def test_host_cost_does_not_grow_with_the_block():
    """Choosing the form takes a few window patterns, not all p^2 of them: a call at p = 64 costs the
    host about what one at p = 4 does (13 us; with all patterns 195).  Best of many, and a
    factor of three for the difference."""
    best = {}
    for p in (4, 64):
        cfg = lbl.config_default("DA_LETKF", 128, 16, ny=128, da_xyprune=p, letkf_rloc_len=1)
        d_in = torch.ones((16, 9, 128, 128), device="cuda") / 9
        out, mac = torch.empty_like(d_in), torch.empty((16, 3, 128, 128), device="cuda")
        yo = torch.zeros((3, 128 // p, 128 // p), device="cuda")
        fn, stream = lbl.load_library().lbl_letkf_analysis_noalloc, torch.cuda.current_stream().cuda_stream
        times = []
        for _ in range(60):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            rc = fn(ctypes.byref(cfg), d_in.data_ptr(), out.data_ptr(), mac.data_ptr(), yo.data_ptr(), stream, None,
                    None, 0)
            times.append(time.perf_counter() - t0)
            assert rc == 0
        torch.cuda.synchronize()
        best[p] = min(times)
    print({p: f"{t * 1e6:.1f} us" for p, t in best.items()})
    assert best[64] < 3 * best[4]
