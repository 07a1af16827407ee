"""lbl_get_fields and lbl_get_ens_stats reduce on the device; their fields equal the host loops of
io.cu:61-139 bit for bit: FP32 central differences, the members added in order, one rounding per
operation.  numpy's float32 arithmetic restates those loops."""
import numpy as np
import pytest

import lbl

pytestmark = pytest.mark.gpu


def _vorticity(u, v, two_dx):
    uy = (np.roll(u, -1, 0) - np.roll(u, 1, 0)) / two_dx
    vx = (np.roll(v, -1, 1) - np.roll(v, 1, 1)) / two_dx
    return vx - uy


@pytest.mark.parametrize("nx,ny,M", [(32, 8, 1), (64, 64, 1), (96, 40, 3), (64, 24, 5), (32, 16, 64)])
def test_accessors_match_the_host_loops(nx, ny, M):
    e = lbl.Ensemble(lbl.config_default("NATURE", nx, M, ny=ny))
    e.init(0)
    e.update(0, 7)
    two_dx = np.float32(2) * (np.float32(e.cfg.h_ref) / np.float32(ny - 1))
    um, vm, wm, w2 = (np.zeros((ny, nx), np.float32) for _ in range(4))
    iv = np.float32(1) / np.float32(M)
    for m in range(M):
        _, u, v, w = e.get_fields(m)
        want = _vorticity(u, v, two_dx)
        np.testing.assert_array_equal(w, want)
        um, vm, wm = um + u, vm + v, wm + want
        w2 = w2 + iv * (want * want)
    um, vm, wm = um * iv, vm * iv, wm * iv
    with np.errstate(invalid="ignore"):
        std = np.sqrt(w2 - wm * wm)
    for got, want in zip(e.ens_stats(), (um, vm, wm, std)):
        assert got.dtype == want.dtype == np.float32
        np.testing.assert_array_equal(got, want)
    e.close()
