"""Calls whose operands or scratch start off 16 bytes where a kernel has a 16-byte path: the path may not be taken, results stay right."""
import ctypes

import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu

NHWC = lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)  # noqa: E731


# channels per group off a multiple of four: the second group's channels start between 16-byte pieces although every pixel is aligned
@pytest.mark.parametrize("variant", ["", "strip"])                     # the tensor-memory kernel, the one with both operands in shared memory
@pytest.mark.parametrize("kernel", [1, 3])
@pytest.mark.parametrize("cig,cog,groups", [(34, 34, 2), (33, 40, 4), (36, 34, 2), (34, 36, 2), (66, 130, 2)])
def test_grouped_channels_last_dweight(cig, cog, groups, kernel, variant, monkeypatch):
    if variant:
        monkeypatch.setenv("B200_DW_VARIANT", variant)
    rng = np.random.default_rng(cig + cog + kernel)
    x, go = (rng.standard_normal((2, c * groups, 12, 13), dtype=np.float32) for c in (cig, cog))
    w, pad = np.zeros((cog * groups, cig, kernel, kernel), np.float32), (kernel // 2,) * 2
    want = oracle.torch_conv_all(x, w, None, go, (1, 1), pad, (1, 1), groups)[2]
    dw = b200conv.conv2d_backward(NHWC(go), NHWC(x), w, padding=pad, groups=groups, mask=(False, True, False), algo="tc")[1]
    assert b200conv.last_kernel() == "tc_strip_dweight" and b200conv.device_status() == 0
    assert oracle.rel_l2(dw, want) <= 1e-5


def _dweight(g, x, go, kw, offset, budget):
    """dWeight through the C ABI with scratch that starts `offset` bytes into its allocation."""
    L, P = b200conv.lib(), ctypes.c_void_p
    p = b200conv.geometry(g.x_shape, g.w_shape[0], g.w_shape[2:], **kw)
    n = b200conv.workspace_bytes(p, b200conv.PHASE_DWEIGHT, budget=budget)
    assert n > 0                                                       # split: the partial sums go through the scratch
    vx, vg, ws, dw = b200conv.DeviceView(x), b200conv.DeviceView(go), b200conv.DeviceBuffer(n + 16), b200conv.DeviceBuffer(4 * int(np.prod(g.w_shape)))
    b200conv.check(L.b200_conv2d_dweight(ctypes.byref(p), vx.view4(), vg.view4(), P(dw.ptr), P(ws.ptr + offset), n, b200conv.ALGO_AUTO, None))
    return dw.to_numpy(g.w_shape)


# one reader of the partial sums for each route: the tensor-memory kernel (3x3), the shared-memory one (1x1, many pixels), grouped
@pytest.mark.parametrize("offset", [4, 8, 12])
@pytest.mark.parametrize("xshape,cout,kernel,kw", [((4, 64, 28, 28), 64, (3, 3), dict(padding=(1, 1))), ((8, 256, 52, 52), 64, (1, 1), dict()),
                                                   ((4, 64, 32, 32), 64, (3, 3), dict(padding=(1, 1), groups=8))], ids=["3x3", "1x1", "grouped"])
def test_dweight_scratch_off_16_bytes(xshape, cout, kernel, kw, offset):
    rng = np.random.default_rng(offset)
    g = oracle.geometry(xshape, cout, kernel, **kw)
    x, go = rng.standard_normal(g.x_shape, dtype=np.float32), rng.standard_normal(g.y_shape, dtype=np.float32)
    want = oracle.torch_conv_all(x, np.zeros(g.w_shape, np.float32), None, go, (1, 1), kw.get("padding", (0, 0)), (1, 1), kw.get("groups", 1))[2]
    got = _dweight(g, x, go, kw, offset, 64 << 20)
    assert b200conv.device_status() == 0 and oracle.rel_l2(got, want) <= 1e-5


@pytest.mark.parametrize("channels,hw", [(512, 7), (64, 28)])          # with the reduction in slices, and whole
@pytest.mark.parametrize("offset", [None, 4])                          # no scratch at all, scratch that is not 16-byte aligned
def test_fused_forward_refuses_unusable_scratch(channels, hw, offset):
    L, P = b200conv.lib(), ctypes.c_void_p
    p = b200conv.geometry((1, channels, hw, hw), channels, (3, 3), padding=(1, 1))
    n = 256 << 20                                                      # as much as the caller says, nothing of it may be touched
    x, w = b200conv.DeviceView(np.zeros((1, channels, hw, hw), np.float32)), b200conv.DeviceView(np.zeros((channels, channels, 3, 3), np.float32))
    y, ws = b200conv.DeviceBuffer(4 * channels * hw * hw), b200conv.DeviceBuffer(16)
    none = b200conv.View4(None, (ctypes.c_int64 * 4)(0, 0, 0, 0))
    scratch = None if offset is None else P(ws.ptr + offset)
    with pytest.raises(b200conv.B200Error, match="workspace"):
        b200conv.check(L.b200_conv2d_forward_fused(ctypes.byref(p), x.view4(), w.view4(), None, 0, none, 1, P(y.ptr), 0, scratch, n, b200conv.ALGO_TC, None))
