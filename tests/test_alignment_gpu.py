"""Calls whose operands or scratch start off 16 bytes where a kernel has a 16-byte path: the path may not be taken, results stay right."""
import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu

NHWC = lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)  # noqa: E731


# channels per group off a multiple of four: the second group's channels start between 16-byte pieces although every pixel is aligned
@pytest.mark.parametrize("variant", ["", "strip"])                     # the tensor-memory kernel, the one with both operands in shared memory
@pytest.mark.parametrize("kernel", [1, 3])
@pytest.mark.parametrize("cig,cog,groups", [(34, 34, 2), (33, 40, 4), (36, 34, 2), (34, 36, 2), (66, 130, 2)])
def test_grouped_channels_last_dweight(cig, cog, groups, kernel, variant, monkeypatch):
    if variant:
        monkeypatch.setenv("B200_DW_VARIANT", variant)
    rng = np.random.default_rng(cig + cog + kernel)
    x, go = (rng.standard_normal((2, c * groups, 12, 13), dtype=np.float32) for c in (cig, cog))
    w, pad = np.zeros((cog * groups, cig, kernel, kernel), np.float32), (kernel // 2,) * 2
    want = oracle.torch_conv_all(x, w, None, go, (1, 1), pad, (1, 1), groups)[2]
    dw = b200conv.conv2d_backward(NHWC(go), NHWC(x), w, padding=pad, groups=groups, mask=(False, True, False), algo="tc")[1]
    assert b200conv.last_kernel() == "tc_strip_dweight" and b200conv.device_status() == 0
    assert oracle.rel_l2(dw, want) <= 1e-5
