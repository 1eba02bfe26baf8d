"""Backward passes of batch norm that keep a tensor in shared memory beside the registers (one wave instead of several), at
the lines of the rule that chooses them and with ragged last units, against the FP64 oracle."""
import numpy as np
import pytest

import b200conv
from oracle import batch_norm_oracle as bn
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
