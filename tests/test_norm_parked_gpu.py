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

# (n, c, h, w), form of the backward pass ("": read again): channels x ranks of four and of five units around a wave of 592 and of 888 CTAs; full threads, one
# unit over, a rank with little; planes that are no whole 16-byte pieces; channels of more values than sixteen CTAs hold
BN = [((5, 593, 32, 32), "parked"), ((5, 888, 32, 32), "parked"), ((5, 704, 30, 34), "parked"), ((64, 256, 14, 14), "parked"), ((64, 297, 14, 14), "registers"),
      ((40, 64, 36, 37), "parked"), ((40, 64, 35, 37), "registers"), ((61, 42, 40, 40), ""), ((62, 40, 36, 36), "")]


@pytest.mark.parametrize("shape,form", BN, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else v or "streamed")
def test_batch_norm(shape, form):
    rng = np.random.default_rng(sum(shape))
    c = shape[1]
    x, g = rng.standard_normal(shape, dtype=np.float32) + np.float32(3), rng.standard_normal(shape, dtype=np.float32)
    w, b = rng.standard_normal(c).astype(np.float32), rng.standard_normal(c).astype(np.float32)
    y, mean, inv = b200conv.batch_norm_forward(x, w, b, None, None, True, 0.1, 1e-5)[:3]
    for training in (True, False):
        second = inv if training else (1 / inv.astype(np.float64) ** 2 - 1e-5).astype(np.float32)
        grads = b200conv.batch_norm_backward(g, x, w, mean, second, training, 1e-5)
        assert b200conv.last_form() == form
        for got, e in zip(grads, bn.backward(g, x, w, mean, second, training, 1e-5, dtype=np.float64)):
            assert oracle.rel_l2(got, e) <= 5 * GATE


# (n, c, h, w), groups, forms forward and backward ("": a CTA reads its row again).  Sixteen CTAs hold 131072 values of a row in registers forward, 65536
# backward (98304 parked), in single values 65536 each; beyond that, shared memory: four CTAs to an SM, then two, up to 409600 values forward and 204800
# backward, less the rounding of sixteen shares.  Eleven ranks; planes cut by ranks and by parts of a warp; a group of 64 planes and, not kept backward, 65.
R, P, S = "registers", "parked", "staged"
GN = [((3, 9, 64, 64), 1, R, R), ((40, 11, 64, 64), 1, R, P), ((20, 96, 22, 66), 32, R, R), ((1, 64, 32, 32), 1, R, R), ((1, 65, 32, 32), 1, R, ""),
      ((1, 24, 64, 64), 1, R, P), ((1, 25, 64, 64), 1, R, S), ((1, 48, 128, 64), 2, S, S), ((1, 32, 64, 64), 1, R, S), ((1, 33, 64, 64), 1, S, S), ((2, 14, 81, 84), 2, R, R),
      ((1, 2, 300, 340), 1, S, ""), ((1, 51, 64, 64), 1, S, ""), ((1, 100, 64, 64), 1, S, ""), ((1, 101, 64, 64), 1, "", ""), ((1, 66, 31, 33), 1, S, ""),
      ((3, 16, 137, 63), 2, S, S), ((1, 4, 227, 225), 1, S, S), ((1, 64, 81, 79), 2, S, S), ((1, 63, 51, 127), 1, S, ""), ((1, 64, 51, 127), 1, "", ""),
      ((2, 5, 1, 1023 * 20), 1, R, S)]


@pytest.mark.parametrize("shape,groups,forward,backward", GN, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else f"g{v}" if isinstance(v, int) else v or "again")
def test_group_norm(shape, groups, forward, backward):
    rng = np.random.default_rng(sum(shape) + groups)
    x, g = rng.standard_normal(shape, dtype=np.float32) + np.float32(30), rng.standard_normal(shape, dtype=np.float32)
    w, b = rng.standard_normal(shape[1]).astype(np.float32), rng.standard_normal(shape[1]).astype(np.float32)
    y, mean, rstd = b200conv.group_norm_forward(x, groups, w, b, 1e-5)
    assert b200conv.last_form() == forward
    wy, wmean, wrstd = gn.forward(x, groups, w, b, 1e-5, dtype=np.float64)
    assert oracle.rel_l2(y, wy) <= 2 * GATE
    np.testing.assert_allclose(mean, wmean, rtol=2e-6, atol=2e-6)
    np.testing.assert_allclose(rstd, wrstd, rtol=1e-5)
    grads = b200conv.group_norm_backward(g, x, mean, rstd, groups, w)
    assert b200conv.last_form() == backward
    for got, e in zip(grads, gn.backward(g, x, mean, rstd, groups, w, dtype=np.float64)):
        assert oracle.rel_l2(got, e) <= 5 * GATE
