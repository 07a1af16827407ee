"""What the host writes to the device is ordered with the kernels that read it.  Contexts and batches run
on non-blocking streams, which do not wait for the legacy stream, and cudaMemcpy from pageable
memory and cudaMemset may return with the device's part still under way there: a batch's table
of pointers read too early is a fault.  Whether it happens depends on the GPU's queues, so the sources
are what is checked: no host-to-device cudaMemcpy and no cudaMemset in the files that use such
streams (the closure's training and inference run on the legacy stream throughout)."""
import os
import re

import pytest

from conftest import PKG


@pytest.mark.parametrize("name", ["lbl_api.cu", "noalloc.cu", "slab.cu", "lbm_kernels.cu", "letkf_kernels.cu",
                                  "letkf_direct.cu", "diag_kernels.cu", "gram_tc.cu", "closure.cu"])
def test_no_legacy_stream_writes(name):
    with open(os.path.join(PKG, "csrc", name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    if name == "closure.cu":
        text = re.search(r"int lbl_set_closure\(.*?\n}\n", text, re.S).group(0)
    bad = re.findall(r"cudaMemcpy\([^;]*cudaMemcpyHostToDevice[^;]*;|cudaMemset\([^;]*;", text)
    assert not bad
