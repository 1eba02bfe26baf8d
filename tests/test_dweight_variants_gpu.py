"""Both tcgen05 dWeight kernels on the geometries that either takes, whichever of them the rule would pick: the layers of
test_dweight_tmem_gpu.py with each kernel pinned, and layers on both sides of the rule that chooses by splits."""
import numpy as np
import pytest

import b200conv
from oracle import oracle
from test_dweight_tmem_gpu import CASES

pytestmark = pytest.mark.gpu

NHWC = lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)  # noqa: E731


# A chain of accumulation has 96 K blocks at most, of 8 truncating steps each, or 12 with three TF32 products.  A step loses 2^-24 * 0.72 on average
# (half a unit in the last place, over the value) of a sum that has reached half of its size on average: 1152 * 2^-25 * 0.72 = 2.5e-5.
GATE = 2.5e-5


def _check(case, layout, budget):
    xshape, cout, kernel, kw = case
    rng = np.random.default_rng(sum(xshape) + cout)
    g = oracle.geometry(xshape, cout, kernel, **kw)
    x, go = rng.standard_normal(g.x_shape, dtype=np.float32), rng.standard_normal(g.y_shape, dtype=np.float32)
    w = np.zeros(g.w_shape, np.float32)
    want = oracle.torch_conv_all(x, w, None, go, kw.get("stride", (1, 1)), kw.get("padding", (0, 0)), kw.get("dilation", (1, 1)), kw.get("groups", 1))[2]
    lay = NHWC if layout == "nhwc" else (lambda a: a)
    dw = b200conv.conv2d_backward(lay(go), lay(x), w, mask=(False, True, False), algo="tc", budget=budget, **kw)[1]
    assert b200conv.last_kernel() == "tc_strip_dweight" and b200conv.device_status() == 0
    assert oracle.rel_l2(dw, want) <= GATE


@pytest.mark.parametrize("variant", ["tmem", "strip"])
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("case", [c for c in CASES if c[0][1] >= 16], ids=lambda c: "x".join(map(str, c[0])) + f"-co{c[1]}-k{c[2][0]}x{c[2][1]}")
def test_pinned(case, layout, variant, monkeypatch):
    monkeypatch.setenv("B200_DW_VARIANT", variant)
    _check(case, layout, 64 << 20)
    _check(case, layout, 0)


# (layer, scratch): few splits and many; 64 and 65 output channels; strips of several phases; 1x1
RULE = [(((7, 16, 21, 21), 62, (3, 3), dict(stride=(2, 2), padding=(1, 1))), 0), (((5, 38, 30, 31), 32, (3, 3), dict(padding=(1, 1))), 0),
        (((6, 40, 40, 40), 64, (3, 3), dict(padding=(1, 1))), 64 << 20), (((5, 38, 30, 31), 65, (3, 3), dict(padding=(1, 1))), 0),
        (((6, 65, 30, 31), 150, (3, 3), dict(stride=(2, 2), padding=(1, 1))), 64 << 20), (((6, 64, 30, 31), 150, (3, 3), dict(stride=(2, 2), padding=(1, 1))), 64 << 20),
        (((9, 48, 20, 20), 40, (1, 1), dict()), 0), (((3, 20, 20, 20), 40, (1, 1), dict()), 0)]


@pytest.mark.parametrize("case,budget", RULE, ids=lambda v: "x".join(map(str, v[0])) + f"-co{v[1]}-k{v[2][0]}" if isinstance(v, tuple) else f"ws{v}")
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
def test_by_rule(case, budget, layout):
    _check(case, layout, budget)
