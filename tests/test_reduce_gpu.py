"""Per-channel and column sums (one launch, cluster-wide): dBias over NCHW, channels-last, sliced and broadcast gradients and
b200_sum_strided's column case, at the edges of their vector width, row batches and cluster ranks, against numpy FP64."""
import ctypes

import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu

# (n, c, h, w): one value, scalar tails, one thread's batch, one pass of a cluster, whole planes off the vector width
SHAPES = [(1, 1, 1, 1), (2, 3, 5, 7), (64, 512, 7, 7), (3, 5, 32, 32), (8, 64, 56, 56), (5, 33, 13, 16), (1, 2, 300, 301), (2, 1040, 4, 4),
          (70, 4, 17, 9), (32, 20, 96, 96)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("layout", ["nchw", "nhwc", "sliced", "nhwc_sliced", "broadcast"])
def test_dbias(shape, layout):
    n, c, h, w = shape
    rng = np.random.default_rng(sum(shape))
    go = rng.standard_normal(shape, dtype=np.float32)
    if layout == "nhwc":
        go = np.ascontiguousarray(go.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)
    elif layout == "sliced":
        parent = np.zeros((n, c + 3, h + 2, w + 5), np.float32)
        parent[:, 2:2 + c, 1:1 + h, 3:3 + w] = go
        go = parent[:, 2:2 + c, 1:1 + h, 3:3 + w]
    elif layout == "nhwc_sliced":
        parent = np.zeros((n, h + 1, w + 2, c + 4), np.float32)
        parent[:, :h, 1:1 + w, 4:] = go.transpose(0, 2, 3, 1)
        go = parent[:, :h, 1:1 + w, 4:].transpose(0, 3, 1, 2)
    elif layout == "broadcast":
        go = np.broadcast_to(go[:, :, :1, :1], shape)
    x, k = np.zeros((n, 1, h, w), np.float32), np.zeros((c, 1, 1, 1), np.float32)
    db = b200conv.conv2d_backward(go, x, k, mask=(False, False, True))[2]
    want = go.astype(np.float64).sum((0, 2, 3))
    scale = np.abs(go.astype(np.float64)).sum((0, 2, 3))
    assert np.all(np.abs(db - want) <= 1e-6 * scale + 1e-12)


@pytest.mark.parametrize("rows,cols,pitch", [(1, 1, 1), (7, 3, 3), (4096, 2048, 2048), (1000, 77, 80), (513, 1000, 1000), (33, 4097, 4100), (20000, 8, 8)])
def test_column_sums(rows, cols, pitch):
    rng = np.random.default_rng(rows + cols)
    a = rng.standard_normal((rows, pitch), dtype=np.float32)
    view = b200conv.DeviceView(a)
    out = b200conv.DeviceBuffer(4 * cols)
    sizes, strides = (ctypes.c_int64 * 2)(rows, cols), (ctypes.c_int64 * 2)(pitch, 1)
    b200conv.check(b200conv.lib().b200_sum_strided(out.ptr, view.ptr, 2, sizes, strides, ctypes.create_string_buffer(b"\x01\x00", 2), None))
    got, want = out.to_numpy((cols,)), a[:, :cols].astype(np.float64).sum(0)
    assert oracle.rel_l2(got, want) <= 1e-6


@pytest.mark.parametrize("n,groups,cpg,h,w", [(1, 2, 4, 3, 3), (2, 3, 8, 5, 33), (5, 4, 4, 17, 40), (3, 2, 8, 64, 31), (16, 2, 4, 32, 32), (9, 32, 8, 9, 65)])
def test_grouped_dweight_tiles(n, groups, cpg, h, w):
    """Row and column tiles with remainders, one tile per block up to many, one block and several blocks per group."""
    rng = np.random.default_rng(n + groups + h + w)
    c = groups * cpg
    x, go = rng.standard_normal((n, c, h, w), dtype=np.float32), rng.standard_normal((n, c, h, w), dtype=np.float32)
    wt = np.zeros((c, cpg, 3, 3), np.float32)
    want = oracle.torch_conv_all(x, wt, None, go, (1, 1), (1, 1), (1, 1), groups)[2]
    for nhwc in (False, True):
        lay = (lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1)).transpose(0, 3, 1, 2)) if nhwc else (lambda a: a)
        dw = b200conv.conv2d_backward(lay(go), lay(x), wt, padding=(1, 1), groups=groups, mask=(False, True, False))[1]
        assert oracle.rel_l2(dw, want) <= 1e-5
