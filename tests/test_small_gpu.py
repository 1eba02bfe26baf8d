"""The one-launch kernel for convolutions of a few tiles: forward, fused forward and dInput where its plan changes (one rank and eight,
pairs of a rank that straddle two channel blocks, ragged channel blocks and column tiles, shares of columns that do not divide a tile),
against PyTorch CPU FP64.  The chains are those of the strip kernels or shorter: held to their 1e-5."""
import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu

CASES = [  # (xshape, cout, kernel, conv arguments)
    ((1, 64, 28, 28), 64, (3, 3), dict(padding=(1, 1))),
    ((1, 16, 5, 6), 16, (1, 1), dict()),                               # one rank, one pair
    ((1, 33, 9, 10), 17, (3, 3), dict(padding=(1, 1))),                # one channel into the second block
    ((2, 256, 7, 7), 40, (3, 3), dict(padding=(1, 1))),                # eight ranks
    ((1, 96, 14, 13), 65, (1, 1), dict()),                             # one channel into the second column tile
    ((1, 160, 12, 11), 32, (2, 3), dict(padding=(0, 1))),              # five blocks of six taps: ranks straddle blocks
    ((1, 32, 20, 40), 48, (3, 3), dict(padding=(2, 2), dilation=(2, 2))),
    ((3, 24, 6, 7), 96, (5, 5), dict(padding=(2, 2))),
    ((1, 512, 7, 7), 64, (1, 1), dict()),
    ((1, 40, 1, 130), 64, (1, 7), dict(padding=(0, 3))),
]


def _lay(a, layout):
    if layout == "nhwc":
        return np.ascontiguousarray(a.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)
    if layout == "view":      # an interior, mirrored
        n, c, h, w = a.shape
        base = np.zeros((n, c + 3, h + 1, w + 3), np.float32)
        base[:, 2:2 + c, 1:, 1:1 + w] = a[:, :, ::-1, ::-1]
        return base[:, 2:2 + c, 1:, 1:1 + w][:, :, ::-1, ::-1]
    return a


@pytest.mark.parametrize("layout", ["nchw", "nhwc", "view"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"-co{c[1]}-k{c[2][0]}x{c[2][1]}")
def test_forward_fused_and_dinput(case, layout):
    xshape, cout, kernel, kw = case
    rng = np.random.default_rng(sum(xshape) + cout)
    g = oracle.geometry(xshape, cout, kernel, **kw)
    x, go = rng.standard_normal(g.x_shape, dtype=np.float32), rng.standard_normal(g.y_shape, dtype=np.float32)
    w = (rng.standard_normal(g.w_shape, dtype=np.float32) / np.sqrt(np.prod(g.w_shape[1:]))).astype(np.float32)
    b, res = rng.standard_normal(cout, dtype=np.float32), rng.standard_normal(g.y_shape, dtype=np.float32)
    y64, dx64 = oracle.torch_conv_all(x, w, b, go, (1, 1), kw.get("padding", (0, 0)), kw.get("dilation", (1, 1)), 1)[:2]

    def one_launch(kernel, call):
        before = b200conv.launch_count()
        out = call()
        assert b200conv.launch_count() == before + 1 and b200conv.last_kernel() == kernel and b200conv.device_status() == 0
        return out
    y = one_launch("tc_small_forward", lambda: b200conv.conv2d_forward(_lay(x, layout), w, b, **kw))
    assert oracle.rel_l2(y, y64) <= 1e-5
    fused = one_launch("tc_small_forward_fused", lambda: b200conv.conv2d_forward_fused(_lay(x, layout), w, b, residual=_lay(res, layout), relu=True, **kw))
    assert oracle.rel_l2(fused, np.maximum(y64 + res, 0)) <= 1e-5
    w_turned = np.ascontiguousarray(w.transpose(1, 0, 2, 3)).transpose(1, 0, 2, 3)      # the filter through other strides
    dx = one_launch("tc_small_dinput", lambda: b200conv.conv2d_backward(_lay(go, layout), x, w_turned, mask=(True, False, False), **kw)[0])
    assert oracle.rel_l2(dx, dx64) <= 1e-5
