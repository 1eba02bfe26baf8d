"""Forward and dInput with the reduction channels in slices: planes off the vector width, strides, dilation, ragged column tiles, strided
filters and residuals, one slice per channel block and several, against PyTorch FP64."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu

CASES = [  # (xshape, cout, k, stride, padding, dilation)
    ((1, 512, 7, 7), 512, 3, 1, 1, 1), ((1, 256, 14, 14), 256, 3, 1, 1, 1), ((2, 128, 28, 28), 128, 3, 1, 1, 1), ((4, 320, 20, 20), 32, 3, 1, 1, 1),
    ((8, 512, 7, 7), 70, 3, 1, 1, 1), ((3, 384, 9, 13), 384, 3, 2, 1, 1), ((2, 192, 11, 10), 200, 3, 1, 2, 2), ((1, 2048, 5, 5), 128, 1, 1, 0, 1),
    ((64, 512, 7, 7), 512, 3, 1, 1, 1), ((1, 160, 16, 16), 256, 3, 1, 1, 1),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
def test_slices(case, layout):
    xshape, cout, k, s, p, d = case
    rng = np.random.default_rng(sum(xshape) + cout)
    r = lambda *shape: rng.standard_normal(shape, dtype=np.float32)
    lay = (lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)) if layout == "nhwc" else (lambda a: a)
    x, w, b = lay(r(*xshape)), lay(r(cout, xshape[1], k, k) * np.float32(0.1)), r(cout)
    args = dict(stride=(s, s), padding=(p, p), dilation=(d, d))
    tx, tw = (torch.from_numpy(np.ascontiguousarray(a)).double() for a in (x, w))
    want = F.conv2d(tx, tw, torch.from_numpy(b).double(), s, p, d)
    res, go = lay(r(*want.shape)), lay(r(*want.shape))
    assert oracle.rel_l2(b200conv.conv2d_forward(x, w, b, algo="tc", **args), want.numpy()) <= 1e-5
    fused = b200conv.conv2d_forward_fused(x, w, b, residual=res, relu=True, algo="tc", **args)
    assert oracle.rel_l2(fused, torch.relu(want + torch.from_numpy(np.ascontiguousarray(res)).double()).numpy()) <= 1e-5
    dx = b200conv.conv2d_backward(go, x, w, mask=(True, False, False), algo="tc", **args)[0]
    wdx = torch.nn.grad.conv2d_input(tx.shape, tw, torch.from_numpy(np.ascontiguousarray(go)).double(), s, p, d)
    assert oracle.rel_l2(dx, wdx.numpy()) <= 1e-5 and b200conv.device_status() == 0
