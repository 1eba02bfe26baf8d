"""Backward passes of the normalisations that keep a tensor in shared memory beside the registers (one wave instead of several, rows that four units a
thread do not hold), at the lines of the rules that choose them and with ragged last units, against the FP64 oracles."""
import numpy as np
import pytest

import b200conv
from oracle import batch_norm_oracle as bn
from oracle import group_norm_oracle as gn
from oracle import oracle

pytestmark = pytest.mark.gpu
GATE = 2e-6

# (n, c, h, w): channels x ranks of four and of five units around a wave of 592 and of 888 CTAs; full threads, one unit over, a rank with little
BN = [(5, 593, 32, 32), (5, 888, 32, 32), (5, 704, 30, 34), (64, 256, 14, 14), (64, 297, 14, 14), (40, 64, 36, 37), (61, 42, 40, 40), (62, 40, 36, 36)]


@pytest.mark.parametrize("shape", BN, ids=lambda s: "x".join(map(str, s)))
def test_batch_norm(shape):
    rng = np.random.default_rng(sum(shape))
    c = shape[1]
    x, g = rng.standard_normal(shape, dtype=np.float32) + np.float32(3), rng.standard_normal(shape, dtype=np.float32)
    w, b = rng.standard_normal(c).astype(np.float32), rng.standard_normal(c).astype(np.float32)
    y, mean, inv = b200conv.batch_norm_forward(x, w, b, None, None, True, 0.1, 1e-5)[:3]
    for training in (True, False):
        second = inv if training else (1 / inv.astype(np.float64) ** 2 - 1e-5).astype(np.float32)
        for got, e in zip(b200conv.batch_norm_backward(g, x, w, mean, second, training, 1e-5), bn.backward(g, x, w, mean, second, training, 1e-5, dtype=np.float64)):
            assert oracle.rel_l2(got, e) <= 5 * GATE


# (n, c, h, w), groups.  Registers hold 65536 values of a row forward and backward 65536 (planes of whole 16-byte pieces; half of them are the gradient's);
# beyond that, shared memory: four CTAs to an SM, sixteen CTAs with two to an SM, the widest row and the first beyond it.  Eleven ranks, one wave with two
# thirds of the ranks; planes cut by ranks and by parts of a warp, a group of 64 planes and of 65.
GN = [((3, 9, 64, 64), 1), ((40, 11, 64, 64), 1), ((20, 96, 22, 66), 32), ((1, 64, 32, 32), 1), ((1, 65, 32, 32), 1), ((1, 24, 64, 64), 1), ((1, 48, 128, 64), 2), ((1, 33, 64, 64), 1),
      ((2, 14, 81, 84), 2), ((1, 2, 300, 340), 1), ((1, 51, 64, 64), 1), ((1, 100, 64, 64), 1), ((1, 101, 64, 64), 1), ((1, 66, 31, 33), 1), ((3, 16, 137, 63), 2),
      ((1, 4, 227, 225), 1), ((1, 64, 81, 79), 2), ((1, 63, 51, 127), 1), ((1, 64, 51, 127), 1), ((2, 5, 1, 1023 * 20), 1)]


@pytest.mark.parametrize("shape,groups", GN, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else f"g{v}")
def test_group_norm(shape, groups):
    rng = np.random.default_rng(sum(shape) + groups)
    x, g = rng.standard_normal(shape, dtype=np.float32) + np.float32(30), rng.standard_normal(shape, dtype=np.float32)
    w, b = rng.standard_normal(shape[1]).astype(np.float32), rng.standard_normal(shape[1]).astype(np.float32)
    y, mean, rstd = b200conv.group_norm_forward(x, groups, w, b, 1e-5)
    wy, wmean, wrstd = gn.forward(x, groups, w, b, 1e-5, dtype=np.float64)
    assert oracle.rel_l2(y, wy) <= 2 * GATE
    np.testing.assert_allclose(mean, wmean, rtol=2e-6, atol=2e-6)
    np.testing.assert_allclose(rstd, wrstd, rtol=1e-5)
    for got, e in zip(b200conv.group_norm_backward(g, x, mean, rstd, groups, w), gn.backward(g, x, mean, rstd, groups, w, dtype=np.float64)):
        assert oracle.rel_l2(got, e) <= 5 * GATE
