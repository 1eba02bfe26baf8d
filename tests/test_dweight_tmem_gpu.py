"""dWeight with the output gradient in tensor memory: the places where its plan changes (half-empty lanes and the shifted second
half, ring wraps, images too wide for a ring that holds every vertical tap, strides and dilations that split a filter row into
strips, ragged channel blocks, accumulation chains cut into several folds, no workspace), against PyTorch CPU FP64."""
import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu

CASES = [  # (xshape, cout, kernel, conv arguments)
    ((2, 32, 20, 20), 64, (3, 3), dict(padding=(1, 1))),                        # 64 output channels: two vertical taps per strip
    ((2, 48, 9, 31), 33, (2, 3), dict(padding=(0, 1))),
    ((1, 40, 23, 17), 64, (5, 5), dict(padding=(2, 2))),                        # five vertical taps: three strips
    ((2, 32, 19, 18), 48, (3, 3), dict(stride=(2, 2), padding=(1, 1))),         # shifted by two taps, column phases
    ((1, 32, 20, 21), 64, (3, 3), dict(padding=(2, 2), dilation=(2, 2))),
    ((2, 64, 12, 13), 65, (3, 3), dict(padding=(1, 1))),                        # one channel into the second half
    ((1, 72, 10, 11), 129, (3, 3), dict(padding=(1, 1))),                       # one channel into the second tile, ragged input block
    ((1, 32, 6, 300), 128, (3, 3), dict(padding=(1, 1))),                       # a wide image: one vertical tap per CTA
    ((3, 160, 7, 7), 96, (3, 3), dict(padding=(1, 1))),                         # rings larger than an image
    ((1, 64, 16, 16), 128, (1, 7), dict(padding=(0, 3))),                       # seven N blocks
    ((1, 64, 16, 16), 128, (7, 1), dict(padding=(3, 0))),
    ((2, 32, 15, 14), 96, (3, 3), dict(stride=(3, 2), padding=(0, 1))),
    ((1, 96, 14, 14), 160, (3, 3), dict(padding=(4, 4), dilation=(4, 4))),      # eight rows between the outer taps
    ((2, 64, 14, 14), 64, (3, 3), dict(padding=(1, 1), groups=2)),
    ((2, 3, 32, 33), 64, (7, 7), dict(stride=(2, 2), padding=(3, 3))),          # filter rows folded into the channels: 21 of 32
    ((1, 8, 19, 20), 130, (5, 5), dict(padding=(2, 2))),                        # 40: two strips
    ((3, 1, 17, 16), 16, (3, 3), dict(padding=(1, 1))),
    ((1, 16, 5, 6), 16, (1, 1), dict()),                                        # 1x1: one K block ...
    ((2, 96, 7, 7), 131, (1, 1), dict()),
    ((3, 300, 9, 8), 40, (1, 1), dict(stride=(2, 2))),
    ((2, 288, 91, 100), 24, (1, 1), dict()),                                    # ... and on either side of the line between the kernels
    ((2, 289, 91, 100), 24, (1, 1), dict()),
    ((2, 15, 12, 13), 40, (3, 3), dict(stride=(1, 3), padding=(0, 1), dilation=(2, 1))),
]


def _run(case, layout, budget=64 << 20, gate=1e-5, flip=None):
    xshape, cout, kernel, kw = case
    rng = np.random.default_rng(sum(xshape) + cout)
    g = oracle.geometry(xshape, cout, kernel, **kw)
    x, go = rng.standard_normal(g.x_shape, dtype=np.float32), rng.standard_normal(g.y_shape, dtype=np.float32)
    w = np.zeros(g.w_shape, np.float32)
    want = oracle.torch_conv_all(x, w, None, go, kw.get("stride", (1, 1)), kw.get("padding", (0, 0)), kw.get("dilation", (1, 1)), kw.get("groups", 1))[2]
    lay = (lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)) if layout == "nhwc" else (lambda a: a)
    mirror = lambda a: lay(np.ascontiguousarray(a[flip]))[flip] if flip else lay(a)  # noqa: E731  the same values through negative strides
    dw = b200conv.conv2d_backward(mirror(go), mirror(x), w, mask=(False, True, False), algo="tc", budget=budget, **kw)[1]
    assert b200conv.last_kernel() == "tc_strip_dweight" and b200conv.device_status() == 0
    assert oracle.rel_l2(dw, want) <= gate


@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"-co{c[1]}-k{c[2][0]}x{c[2][1]}")
def test_dweight(case, layout):
    _run(case, layout)


_BACK, _ALL = slice(None, None, -1), slice(None)


@pytest.mark.parametrize("flip", [(_BACK,), (_ALL, _ALL, _BACK), (_ALL, _ALL, _ALL, _BACK), (_ALL, _BACK), (_BACK, _ALL, _BACK, _BACK)],
                         ids=["images", "rows", "columns", "channels", "images-rows-columns"])
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("case", [CASES[0], CASES[5], CASES[14], CASES[18]], ids=lambda c: "x".join(map(str, c[0])))
def test_views_with_negative_strides(case, layout, flip):
    _run(case, layout, flip=flip)


@pytest.mark.parametrize("case", [CASES[0], CASES[5], CASES[7]], ids=lambda c: "x".join(map(str, c[0])))
def test_dweight_in_several_folds_and_without_workspace(case, monkeypatch):
    monkeypatch.setenv("B200_DW_CHUNK_KB", "3")     # accumulation chains of three K blocks
    _run(case, "nchw")
    _run(case, "nchw", budget=0)                    # a single split that writes dW itself


# Layers of fewer than 32 (input channel, tap) pairs were computed in FP32 before: short chains.  A chain of four K blocks is 32 truncating steps,
# each of which loses 2^-24 * 0.72 of a sum that has reached half of its size on average: 7e-7; the cross terms' BF16 operands 2^-11 * 2^-9 / sqrt(3)
# of the result twice over: 8e-7 together.
@pytest.mark.parametrize("case", [((12, 3, 60, 61), 80, (3, 3), dict(padding=(1, 1))), ((8, 1, 90, 33), 33, (5, 5), dict(padding=(2, 2), stride=(2, 1))),
                                  ((6, 30, 40, 41), 72, (1, 1), dict()), ((1, 16, 9, 9), 16, (1, 1), dict())], ids=lambda c: "x".join(map(str, c[0])))
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
def test_few_products_keep_fp32(case, layout):
    _run(case, layout, gate=1.2e-6)
    _run(case, layout, budget=0, gate=1.2e-6)
