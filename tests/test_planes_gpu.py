"""1x1 convolutions on whole NCHW planes with the filter kept in shared memory: one to eight channel blocks, the last ragged, each column
tile width and a ragged one, images that end inside a tile and inside a 16-byte piece, a sliced batch, against PyTorch CPU FP64.  Beside them what the
rule leaves to the strip kernel: filters beyond shared memory, column tiles half empty, planes that start off 16 bytes."""
import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu
PLANES, STRIP = "tc_planes_", "tc_strip_"


def _laid_out(a, layout):
    n, c, h, w = a.shape
    if layout == "sliced":                # the channels 4 .. of a wider tensor
        base = np.zeros((n, c + 8, h, w), np.float32)
        base[:, 4:-4] = a
        return base[:, 4:-4]
    if layout == "padded":                # planes of h * w pixels at multiples of four floats: the last piece of a line is partly another's
        base = np.full((n, c, -(-h * w // 4) * 4), np.nan, np.float32)
        base[:, :, :h * w] = a.reshape(n, c, h * w)
        return np.lib.stride_tricks.as_strided(base, a.shape, (*base.strides[:2], 4 * w, 4))
    return a


def _check(n, cin, cout, h, w, layout, forward, dinput):
    rng = np.random.default_rng(n + cin + cout + h)
    x, go = rng.standard_normal((n, cin, h, w), dtype=np.float32), rng.standard_normal((n, cout, h, w), dtype=np.float32)
    wt = (rng.standard_normal((cout, cin, 1, 1), dtype=np.float32) / np.sqrt(cin)).astype(np.float32)
    b = rng.standard_normal(cout, dtype=np.float32)
    y64, dx64 = oracle.torch_conv_all(x, wt, b, go, (1, 1), (0, 0), (1, 1), 1)[:2]
    y = b200conv.conv2d_forward(_laid_out(x, layout), wt, b, algo="tc")
    assert b200conv.last_kernel() == forward + "forward" and b200conv.device_status() == 0 and oracle.rel_l2(y, y64) <= 1e-5
    dx = b200conv.conv2d_backward(_laid_out(go, layout), x, wt, mask=(True, False, False), algo="tc")[0]
    assert b200conv.last_kernel() == dinput + "dinput" and b200conv.device_status() == 0 and oracle.rel_l2(dx, dx64) <= 1e-5


@pytest.mark.parametrize("n,cin,cout,h,w,forward,dinput", [
    (60, 256, 64, 24, 22, PLANES, PLANES), (75, 32, 33, 16, 33, PLANES, PLANES), (64, 40, 33, 26, 30, PLANES, PLANES), (64, 64, 256, 28, 28, PLANES, PLANES),
    (60, 128, 100, 22, 26, PLANES, PLANES), (60, 33, 200, 24, 24, PLANES, PLANES), (1, 64, 64, 195, 196, PLANES, PLANES),
    (64, 32, 48, 84, 84, PLANES, PLANES),      # two dozen tiles to a CTA: every accumulator is used again and again
    (75, 16, 16, 16, 33, STRIP, STRIP),        # less than half a column tile
    (60, 288, 64, 24, 22, STRIP, STRIP),       # nine channel blocks of 16 KB; two column tiles
])
@pytest.mark.parametrize("sliced", [False, True])
def test_forward_and_dinput(n, cin, cout, h, w, forward, dinput, sliced):
    _check(n, cin, cout, h, w, "sliced" if sliced else "dense", forward, dinput)


# planes whose number of pixels is no multiple of four: dense ones start off 16 bytes, padded ones end inside a piece
@pytest.mark.parametrize("n,cin,cout,h,w", [(60, 64, 48, 23, 23), (75, 32, 64, 19, 31), (64, 40, 100, 25, 27)])
@pytest.mark.parametrize("layout", ["dense", "padded"])
def test_planes_that_end_inside_a_piece(n, cin, cout, h, w, layout):
    name = PLANES if layout == "padded" else STRIP
    _check(n, cin, cout, h, w, layout, name, name)
