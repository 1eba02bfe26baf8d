"""Fused attention (scores never in memory): edges of its 128-row tiles and 64-column blocks, one block and many, ragged head
dimensions, causal tiles on and off the diagonal, scores that make the running maximum move, against the FP64 oracle."""
import numpy as np
import pytest

import b200conv
from oracle import attention_oracle as att
from oracle import oracle

pytestmark = pytest.mark.gpu

CASES = [  # (batch, tq, tk, d, causal)
    (1, 32, 32, 16, False), (2, 128, 64, 64, False), (1, 129, 65, 64, False), (3, 100, 77, 40, False), (2, 64, 1000, 32, False),
    (1, 300, 300, 64, True), (2, 257, 257, 33, True), (1, 90, 400, 64, True), (1, 400, 90, 48, True), (5, 511, 513, 64, False),
    (160, 64, 77, 32, False),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
@pytest.mark.parametrize("spread", [1.0, 6.0])     # 6: row maxima that grow by tens from block to block
def test_fused(case, spread):
    batch, tq, tk, d, causal = case
    rng = np.random.default_rng(sum(case[:4]))
    r = lambda *s: rng.standard_normal(s, dtype=np.float32)
    q, k, v, grad = r(batch, tq, d) * np.float32(spread), r(batch, tk, d), r(batch, tk, d), r(batch, tq, d)
    out, lse = b200conv.attention_forward(q, k, v, None, causal)
    assert b200conv.last_kernel() == "attention_forward: fused"
    wout, wlse = att.forward(q, k, v, None, causal)
    assert oracle.rel_l2(out, wout) <= 2e-5
    np.testing.assert_allclose(lse, wlse, rtol=1e-5, atol=2e-5)
    got = b200conv.attention_backward(grad, q, k, v, out, lse, None, causal)
    assert b200conv.last_kernel() == "attention_backward: fused" and b200conv.device_status() == 0
    for a, b in zip(got, att.backward(grad, q, k, v, wout, wlse, None, causal)):
        assert oracle.rel_l2(a, b) <= 5e-5
