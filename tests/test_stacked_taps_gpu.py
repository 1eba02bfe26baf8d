"""Forward and dInput with 64 or fewer result channels in the transposed strip kernel, two filter taps to a tile: odd and even filter widths,
dilations (the stacked taps lie that far apart), strides (neighbours within a phase), ragged channel blocks, images smaller than a tile and
tiles that end inside one, groups, against PyTorch CPU FP64."""
import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu

CASES = [  # (xshape, cout, kernel, conv arguments)
    ((2, 64, 20, 20), 64, (3, 3), dict(padding=(1, 1))),
    ((1, 16, 5, 6), 16, (3, 3), dict(padding=(1, 1))),
    ((3, 40, 23, 17), 33, (3, 3), dict(padding=(2, 2), dilation=(2, 2))),
    ((2, 48, 9, 31), 50, (2, 2), dict(padding=(0, 1))),
    ((1, 32, 19, 100), 32, (5, 5), dict(padding=(2, 2))),          # (four rows of 102 pixels beside a tile still fit shared memory)
    ((2, 33, 31, 30), 64, (3, 3), dict(stride=(2, 2), padding=(1, 1))),
    ((1, 32, 40, 41), 64, (1, 7), dict(padding=(0, 3))),
    ((2, 96, 14, 15), 96, (3, 3), dict(padding=(1, 1), groups=3)),
    ((9, 64, 56, 56), 64, (3, 3), dict(padding=(1, 1))),
    ((1, 64, 12, 40), 48, (3, 3), dict(padding=(0, 16), dilation=(1, 16))),
]


@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"-co{c[1]}-k{c[2][0]}x{c[2][1]}")
def test_forward_and_dinput(case, layout, monkeypatch):
    monkeypatch.setenv("B200_CONV_TC_VARIANT", "stacked")
    xshape, cout, kernel, kw = case
    rng = np.random.default_rng(sum(xshape) + cout)
    g = oracle.geometry(xshape, cout, kernel, **kw)
    x, go = rng.standard_normal(g.x_shape, dtype=np.float32), rng.standard_normal(g.y_shape, dtype=np.float32)
    w = (rng.standard_normal(g.w_shape, dtype=np.float32) / np.sqrt(np.prod(g.w_shape[1:]))).astype(np.float32)
    b = rng.standard_normal(cout, dtype=np.float32)
    y64, dx64 = oracle.torch_conv_all(x, w, b, go, kw.get("stride", (1, 1)), kw.get("padding", (0, 0)), kw.get("dilation", (1, 1)), kw.get("groups", 1))[:2]
    lay = (lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)) if layout == "nhwc" else (lambda a: a)
    y = b200conv.conv2d_forward(lay(x), w, b, **kw)
    assert b200conv.last_kernel() == "tc_strip_forward" and b200conv.device_status() == 0 and oracle.rel_l2(y, y64) <= 1e-5
    dx = b200conv.conv2d_backward(lay(go), lay(x), w, mask=(True, False, False), **kw)[0]
    assert b200conv.last_kernel() == "tc_strip_dinput" and b200conv.device_status() == 0 and oracle.rel_l2(dx, dx64) <= 1e-5
