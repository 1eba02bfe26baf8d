"""Activation views whose channels lie further apart than 32-bit element offsets reach (a tensor held channel first with many pixels, or a slice of one):
forward and dInput of the transposed strip kernel, most of a tile's rows real channels and two taps to a tile, against PyTorch CPU FP64."""
import ctypes

import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu
STRIDE = 150_000_000      # 15 of them are beyond 2^31 elements; 16 channels take 9.6 GB


@pytest.fixture(scope="module")
def far():
    import torch
    if torch.cuda.mem_get_info()[0] < 12 << 30:
        pytest.skip("needs 10 GB of free device memory")
    return torch.empty(15 * STRIDE + 4096, device="cuda")


@pytest.mark.parametrize("wide", [80, 48], ids=["full", "stacked"])     # result channels
@pytest.mark.parametrize("is_dx", [False, True], ids=["forward", "dinput"])
def test_channels_beyond_32_bit_offsets(far, wide, is_dx, monkeypatch):
    import torch
    monkeypatch.setenv("B200_CONV_TC_VARIANT", "tstrip" if wide > 64 else "stacked")
    b200conv.init()
    rng = np.random.default_rng(wide)
    cin, cout = (wide, 16) if is_dx else (16, wide)
    p = b200conv.geometry((1, cin, 20, 20), cout, (3, 3), padding=(1, 1))
    x, go = rng.standard_normal((1, cin, 20, 20), dtype=np.float32), rng.standard_normal((1, cout, 20, 20), dtype=np.float32)
    w = (rng.standard_normal((cout, cin, 3, 3), dtype=np.float32) / np.sqrt(9 * cin)).astype(np.float32)
    act = far.as_strided((1, 16, 20, 20), (16 * STRIDE, STRIDE, 20, 1))
    act.copy_(torch.from_numpy(go if is_dx else x))
    wd, out = torch.from_numpy(w).cuda(), torch.empty(1, wide, 20, 20, device="cuda")
    phase = b200conv.PHASE_DINPUT if is_dx else b200conv.PHASE_FORWARD
    ws_n = b200conv.workspace_bytes(p, phase)
    ws = torch.empty(max(ws_n, 16), dtype=torch.uint8, device="cuda")
    view = lambda t: b200conv.View4(t.data_ptr(), (ctypes.c_int64 * 4)(*t.stride()))  # noqa: E731
    torch.cuda.synchronize()
    if is_dx:
        b200conv.check(b200conv.lib().b200_conv2d_dinput(ctypes.byref(p), view(act), view(wd), out.data_ptr(), ws.data_ptr(), ws_n, 0, None))
    else:
        b200conv.check(b200conv.lib().b200_conv2d_forward(ctypes.byref(p), view(act), view(wd), None, 0, out.data_ptr(), ws.data_ptr(), ws_n, 0, None))
    torch.cuda.synchronize()
    want = oracle.torch_conv_all(x, w, None, go, (1, 1), (1, 1), (1, 1), 1)[1 if is_dx else 0]
    assert b200conv.device_status() == 0 and oracle.rel_l2(out.cpu().numpy(), want) <= 1e-5
