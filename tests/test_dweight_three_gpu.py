"""dWeight of 1x1 filters with 64 or fewer output channels: three TF32 products, the cross terms in accumulators of their own, against FP64.  One
channel block to six (the most that leave room for both accumulators) and beyond, ragged ones, strides, accumulation in several folds, no scratch.

The gate.  The parts of a split operand keep 21 bits: a product is off by up to 2^-21, on average by a quarter of that (1.2e-7), with either sign.  The
tensor core cuts its accumulator after every eight pixels, half a unit in the last place on average (4.3e-8 of the sum so far, which for values of
either sign grows with the square root of their number: two thirds of that of the whole); folds and splits add in FP32.  Cross terms in BF16 are 5e-7 above it for
sums of up to 150 pixels (36 pixels: 1.5e-7 against 7.4e-7, gate 2.6e-7).
"""
import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu


def _error(xshape, cout, stride, layout, budget):
    rng = np.random.default_rng(sum(xshape) + cout)
    g = oracle.geometry(xshape, cout, (1, 1), stride=stride)
    x, go, w = rng.standard_normal(g.x_shape, dtype=np.float32), rng.standard_normal(g.y_shape, dtype=np.float32), np.zeros(g.w_shape, np.float32)
    xs = x.astype(np.float64)[:, :, ::stride[0], ::stride[1]]
    want = np.einsum("nohw,nchw->oc", go.astype(np.float64), xs)[:, :, None, None]
    lay = (lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)) if layout == "nhwc" else (lambda a: a)
    dw = b200conv.conv2d_backward(lay(go), lay(x), w, stride=stride, mask=(False, True, False), budget=budget)[1]
    assert b200conv.last_kernel() == "tc_strip_dweight" and b200conv.device_status() == 0
    return oracle.rel_l2(dw, want)


def _gate(pixels, chain):
    return 1.2e-7 + 4.3e-8 * 2 / 3 * -(-min(pixels, chain) // 8) + (1e-7 if pixels > chain else 0)


@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("xshape,cout,stride", [((1, 384, 7, 7), 56, (1, 1)), ((1, 128, 12, 12), 62, (2, 2)), ((2, 96, 8, 8), 23, (1, 1)), ((1, 32, 7, 9), 64, (1, 1)),
                                                ((1, 33, 9, 9), 16, (1, 1)), ((2, 192, 7, 9), 33, (1, 1)), ((1, 223, 11, 12), 64, (1, 1)), ((3, 416, 13, 7), 48, (2, 1))],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_few_pixels(xshape, cout, stride, layout):
    pixels = xshape[0] * -(-xshape[2] // stride[0]) * -(-xshape[3] // stride[1])
    assert _error(xshape, cout, stride, layout, 64 << 20) <= _gate(pixels, 3072)


@pytest.mark.parametrize("budget", [64 << 20, 0])
@pytest.mark.parametrize("chain", [None, "3"])
@pytest.mark.parametrize("xshape,cout", [((3, 192, 31, 33), 64), ((2, 72, 40, 39), 40), ((5, 256, 23, 21), 17)], ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_longer_sums(xshape, cout, chain, budget, monkeypatch):
    if chain:
        monkeypatch.setenv("B200_DW_CHUNK_KB", chain)
    assert _error(xshape, cout, (1, 1), "nchw", budget) <= _gate(xshape[0] * xshape[2] * xshape[3], 32 * int(chain or 96))
