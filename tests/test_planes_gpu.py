"""1x1 convolutions on whole NCHW planes with the filter kept in shared memory: one to eight channel blocks, the last ragged, each column
tile width and a ragged one, images that end inside a tile and inside a 16-byte piece's line, a sliced batch, against PyTorch CPU FP64."""
import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cin,cout,h,w", [
    (60, 256, 64, 24, 22), (75, 16, 16, 16, 33), (64, 40, 33, 26, 30), (64, 64, 256, 28, 28), (60, 128, 100, 22, 26), (60, 33, 200, 24, 24),
    (1, 64, 64, 195, 196),
    (64, 32, 48, 84, 84),      # two dozen tiles to a CTA: every accumulator is used again and again
])
@pytest.mark.parametrize("sliced", [False, True])
def test_forward_and_dinput(n, cin, cout, h, w, sliced):
    rng = np.random.default_rng(n + cin + cout + h)
    x, go = rng.standard_normal((n, cin, h, w), dtype=np.float32), rng.standard_normal((n, cout, h, w), dtype=np.float32)
    wt = (rng.standard_normal((cout, cin, 1, 1), dtype=np.float32) / np.sqrt(cin)).astype(np.float32)
    b = rng.standard_normal(cout, dtype=np.float32)
    y64, dx64 = oracle.torch_conv_all(x, wt, b, go, (1, 1), (0, 0), (1, 1), 1)[:2]

    def view(a):      # the channels 4 .. of a wider tensor
        if not sliced:
            return a
        base = np.zeros((a.shape[0], a.shape[1] + 8, h, w), np.float32)
        base[:, 4:-4] = a
        return base[:, 4:-4]
    y = b200conv.conv2d_forward(view(x), wt, b, algo="tc")
    assert b200conv.device_status() == 0 and oracle.rel_l2(y, y64) <= 1e-5
    dx = b200conv.conv2d_backward(view(go), x, wt, mask=(True, False, False), algo="tc")[0]
    assert b200conv.device_status() == 0 and oracle.rel_l2(dx, dx64) <= 1e-5
