"""Forward passes of layers with fewer than sixteen input channels on the tcgen05 row kernel (im2col rows in tensor memory): edges of
its 128-pixel tiles, its 32-wide K blocks, its column tiles and of the image, against PyTorch CPU FP64."""
import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xshape,cout,kernel,kw", [
    ((2, 3, 32, 32), 64, (7, 7), dict(stride=(2, 2), padding=(3, 3))),       # K = 147: five K blocks, the last one ragged
    ((1, 1, 16, 8), 16, (3, 3), dict(padding=(1, 1))),                       # one tile of 128 pixels exactly, K = 9
    ((1, 1, 43, 3), 17, (1, 1), dict()),                                     # 129 pixels, K = 1
    ((3, 4, 9, 11), 320, (3, 3), dict(padding=(1, 1))),                      # three column tiles, K = 36
    ((2, 8, 17, 23), 130, (3, 3), dict(padding=(1, 1))),                     # two column tiles with two columns to spare
    ((1, 15, 20, 20), 128, (3, 3), dict(padding=(2, 2), dilation=(2, 2))),   # K = 135
    ((2, 2, 30, 31), 48, (4, 5), dict(stride=(3, 2), padding=(0, 2))),
    ((1, 3, 5, 5), 32, (7, 7), dict(padding=(3, 3))),                        # image smaller than the filter
    ((2, 12, 12, 12), 40, (5, 5), dict()),                                   # valid convolution, K = 300
    ((40, 3, 33, 33), 96, (3, 3), dict(stride=(2, 2), padding=(1, 1))),      # more tiles than SMs
], ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v) if isinstance(v, int) else "")
@pytest.mark.parametrize("layout", ["nchw", "nhwc", "sliced"])
def test_narrow_forward(xshape, cout, kernel, kw, layout):
    rng = np.random.default_rng(sum(xshape) + cout)
    g = oracle.geometry(xshape, cout, kernel, **kw)
    x = rng.standard_normal(g.x_shape, dtype=np.float32)
    w = (rng.standard_normal(g.w_shape, dtype=np.float32) / np.sqrt(np.prod(g.w_shape[1:]))).astype(np.float32)
    b = rng.standard_normal(cout, dtype=np.float32)
    want = oracle.torch_conv_all(x, w, b, np.zeros(g.y_shape, np.float32), kw.get("stride", (1, 1)), kw.get("padding", (0, 0)),
                                 kw.get("dilation", (1, 1)), 1)[0]
    if layout == "nhwc":
        x = np.ascontiguousarray(x.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)
    elif layout == "sliced":
        n, c, h, wd = x.shape
        parent = np.zeros((n, c + 3, h + 2, wd + 5), np.float32)
        parent[:, 2:2 + c, 1:1 + h, 3:3 + wd] = x
        x = parent[:, 2:2 + c, 1:1 + h, 3:3 + wd]
    y = b200conv.conv2d_forward(x, w, b, algo="tc", **kw)
    assert b200conv.last_kernel() == "tc_rows_forward" and b200conv.device_status() == 0
    assert oracle.rel_l2(y, want) <= 1e-5
    assert oracle.rel_l2(b200conv.conv2d_forward(x, w, None, algo="tc", **kw), want - b[None, :, None, None]) <= 1e-5


# The layers of this kernel were computed in FP32 on the CUDA cores before it.  Its main products add up in chains of at most 48 truncating
# steps, each of which loses half a unit in the last place on average, 2^-24, of a sum that has reached half of its size on average:
# 48 * 2^-25 * 0.72 (the mean of a unit in the last place over the value) = 1.0e-6 at most; the split itself stays below 2e-7.
@pytest.mark.parametrize("xshape,cout,kernel,kw", [
    ((2, 3, 64, 64), 64, (7, 7), dict(stride=(2, 2), padding=(3, 3))),       # six K blocks, one chain
    ((1, 14, 21, 21), 82, (5, 5), dict(padding=(2, 2))),                     # eighteen: two chains
    ((2, 15, 19, 18), 130, (7, 7), dict(padding=(3, 3))),                    # twenty-seven: three chains, two column tiles
    ((1, 11, 24, 24), 16, (7, 1), dict(padding=(3, 0))),
    ((40, 1, 30, 30), 48, (3, 3), dict(padding=(1, 1))),                     # several tiles per CTA
], ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v) if isinstance(v, int) else "")
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
def test_narrow_forward_keeps_fp32(xshape, cout, kernel, kw, layout):
    rng = np.random.default_rng(sum(xshape) + cout)
    g = oracle.geometry(xshape, cout, kernel, **kw)
    x, b = rng.standard_normal(g.x_shape, dtype=np.float32), rng.standard_normal(cout, dtype=np.float32)
    w = (rng.standard_normal(g.w_shape, dtype=np.float32) / np.sqrt(np.prod(g.w_shape[1:]))).astype(np.float32)
    want = oracle.torch_conv_all(x, w, b, np.zeros(g.y_shape, np.float32), kw.get("stride", (1, 1)), kw.get("padding", (0, 0)), (1, 1), 1)[0]
    if layout == "nhwc":
        x = np.ascontiguousarray(x.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)
    y = b200conv.conv2d_forward(x, w, b, algo="tc", **kw)
    assert b200conv.last_kernel() == "tc_rows_forward" and b200conv.device_status() == 0
    assert oracle.rel_l2(y, want) <= 1.2e-6
