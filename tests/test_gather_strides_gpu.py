"""The gather dWeight kernel (filters wider than eight taps) on views with negative strides, against PyTorch CPU FP64."""
import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu
_BACK, _ALL = slice(None, None, -1), slice(None)


@pytest.mark.parametrize("flip", [(_BACK,), (_ALL, _BACK), (_ALL, _ALL, _BACK), (_ALL, _ALL, _ALL, _BACK), (_BACK, _BACK, _BACK, _BACK)],
                         ids=["images", "channels", "rows", "columns", "all"])
@pytest.mark.parametrize("groups", [1, 2])
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
def test_dweight(layout, groups, flip):
    rng = np.random.default_rng(groups)
    kw = dict(padding=(0, 4), groups=groups)
    g = oracle.geometry((2, 32 * groups, 5, 17), 32 * groups, (1, 9), **kw)
    x, go = rng.standard_normal(g.x_shape, dtype=np.float32), rng.standard_normal(g.y_shape, dtype=np.float32)
    w = np.zeros(g.w_shape, np.float32)
    want = oracle.torch_conv_all(x, w, None, go, (1, 1), (0, 4), (1, 1), groups)[2]
    lay = (lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)) if layout == "nhwc" else (lambda a: a)
    view = lambda a: lay(np.ascontiguousarray(a[flip]))[flip]  # noqa: E731  the same values through negative strides
    dw = b200conv.conv2d_backward(view(go), view(x), w, mask=(False, True, False), algo="tc", **kw)[1]
    assert b200conv.last_kernel() == "tc_igemm_dweight" and b200conv.device_status() == 0
    assert oracle.rel_l2(dw, want) <= 1e-5
