"""Forward and dInput with 64 or fewer result channels in the transposed strip kernel, two filter taps to a tile: odd and even filter widths,
dilations (the stacked taps lie that far apart), strides (neighbours within a phase, and phases without any), ragged channel blocks, images smaller
than a tile and tiles that end inside one, groups, against PyTorch CPU FP64."""
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
    ((2, 33, 31, 30), 64, (3, 3), dict(stride=(2, 2), padding=(1, 1))),    # columns 0 and 2 in one phase, 1 alone in the other
    ((1, 32, 40, 41), 64, (1, 7), dict(padding=(0, 3))),
    ((2, 96, 14, 15), 96, (3, 3), dict(padding=(1, 1), groups=3)),
    ((9, 64, 56, 56), 64, (3, 3), dict(padding=(1, 1))),
    ((1, 64, 12, 40), 48, (3, 3), dict(padding=(0, 16), dilation=(1, 16))),
    ((2, 32, 13, 21), 32, (3, 5), dict(padding=(1, 2), stride=(1, 2))),       # columns 0, 2, 4 and 1, 3
    ((1, 20, 21, 23), 17, (1, 3), dict(padding=(0, 1))),                      # a stack and a lone tap; one channel on the second warp
    ((3, 50, 25, 28), 48, (3, 3), dict(padding=(1, 1), stride=(2, 1))),
]


def _kernels(case):
    """The kernels of forward and dInput, which is not stacked in several phases."""
    return "tc_stacked_forward", "tc_stacked_dinput" if case[3].get("stride", (1, 1)) == (1, 1) else "tc_strip_dinput"


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
    assert b200conv.last_kernel() == _kernels(case)[0] and b200conv.device_status() == 0 and oracle.rel_l2(y, y64) <= 1e-5
    dx = b200conv.conv2d_backward(lay(go), lay(x), w, mask=(True, False, False), **kw)[0]
    assert b200conv.last_kernel() == _kernels(case)[1] and b200conv.device_status() == 0 and oracle.rel_l2(dx, dx64) <= 1e-5


@pytest.mark.parametrize("case", [*CASES[:8], *CASES[9:]],
                         ids=lambda c: "x".join(map(str, c[0])) + f"-co{c[1]}-k{c[2][0]}x{c[2][1]}")
def test_values_that_are_not_finite_stay_where_the_filter_reaches(case, monkeypatch):
    monkeypatch.setenv("B200_CONV_TC_VARIANT", "stacked")
    xshape, cout, kernel, kw = case
    rng = np.random.default_rng(sum(xshape) + cout)
    g = oracle.geometry(xshape, cout, kernel, **kw)
    x, go = rng.standard_normal(g.x_shape, dtype=np.float32), rng.standard_normal(g.y_shape, dtype=np.float32)
    w = (rng.standard_normal(g.w_shape, dtype=np.float32) / np.sqrt(np.prod(g.w_shape[1:]))).astype(np.float32)
    args = (kw.get("stride", (1, 1)), kw.get("padding", (0, 0)), kw.get("dilation", (1, 1)), kw.get("groups", 1))
    where = {}
    for name, a in (("x", x), ("go", go)):      # a corner, the ends of a row and of the next, and an interior pixel of the last image
        h, wd = a.shape[2:]
        marks = np.zeros_like(a)
        for i, (y0, x0) in enumerate([(0, 0), (h // 2, wd - 1), (h // 2 + 1, 0), (h - 1, wd // 2), (h // 3, wd // 3)]):
            marks[-1, i % a.shape[1], y0, x0] = 1
        where[name] = marks
    reached = oracle.torch_conv_all(where["x"], np.ones_like(w), None, where["go"], *args)[:2]
    want = oracle.torch_conv_all(np.where(where["x"] > 0, 0, x), w, None, np.where(where["go"] > 0, 0, go), *args)[:2]
    for value in (np.inf, np.nan):
        xv, gv = np.where(where["x"] > 0, np.float32(value), x), np.where(where["go"] > 0, np.float32(value), go)
        y = b200conv.conv2d_forward(xv, w, None, **kw)
        assert b200conv.last_kernel() == _kernels(case)[0]
        dx = b200conv.conv2d_backward(gv, xv, w, mask=(True, False, False), **kw)[0]
        assert b200conv.last_kernel() == _kernels(case)[1]
        for a, r, e in zip((y, dx), reached, want):
            assert np.array_equal(np.isfinite(a), r < 0.5)
            assert oracle.rel_l2(np.where(r < 0.5, a, 0), np.where(r < 0.5, e, 0)) <= 1e-5


# kernel of the automatic choice: the stacked form where the models of both kernels say so
@pytest.mark.parametrize("xshape,cout,kernel", [((8, 64, 56, 56), 64, "tc_stacked_forward"), ((16, 32, 33, 33), 64, "tc_strip_forward"), ((8, 64, 56, 56), 65, "tc_tstrip_forward")],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_automatic_choice(xshape, cout, kernel, monkeypatch):
    monkeypatch.delenv("B200_CONV_TC_VARIANT", raising=False)
    rng = np.random.default_rng(cout)
    p = b200conv.geometry(xshape, cout, (3, 3), padding=(1, 1))
    x, w = rng.standard_normal(xshape, dtype=np.float32), (rng.standard_normal((cout, xshape[1], 3, 3), dtype=np.float32) / 24).astype(np.float32)
    want = oracle.torch_conv_all(x, w, None, np.zeros((p.n, p.cout, p.oh, p.ow), np.float32), (1, 1), (1, 1), (1, 1), 1)[0]
    for budget, name in ((b200conv.workspace_bytes(p, b200conv.PHASE_FORWARD), kernel), (0, "simt_igemm_forward")):
        y = b200conv.conv2d_forward(x, w, None, padding=(1, 1), budget=budget)
        assert b200conv.last_kernel() == name and b200conv.device_status() == 0 and oracle.rel_l2(y, want) <= 1e-5
