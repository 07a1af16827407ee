"""The accessors report their own calls' errors, not an earlier one's."""
import numpy as np
import pytest

import lbl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("read", ["fields", "ens_stats"])
def test_accessors_after_a_context_on_a_missing_device(read):
    """A context cannot be made on a device that is not there; the refusal leaves the thread's last CUDA
    error behind.  Another context's fields are none the worse for it."""
    e = lbl.Ensemble(lbl.config_default("NATURE", 64, 2))
    e.init(0)
    e.update(0, 3)
    call = (lambda: e.get_fields(1)) if read == "fields" else e.ens_stats
    before = call()
    with pytest.raises(lbl.LblError):
        lbl.Ensemble(lbl.config_default("NATURE", 64, 2), device=63)
    for a, b in zip(before, call()):
        np.testing.assert_array_equal(a, b)
    e.close()
