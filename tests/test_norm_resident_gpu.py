"""Normalisation rows held in registers by the CTAs of a cluster: one value, one CTA, shares cut inside a plane, empty shares,
planes off the vector width, the largest row that fits and the first that does not, against the FP64 oracles."""
import numpy as np
import pytest

import b200conv
from oracle import batch_norm_oracle as bn
from oracle import group_norm_oracle as gn
from oracle import oracle

pytestmark = pytest.mark.gpu
GATE = 2e-6

# (n, c, h, w) of batch norm: units per channel against threads x units x ranks
BN = [(1, 3, 1, 5), (2, 5, 16, 16), (3, 4, 31, 33), (9, 16, 7, 7), (64, 16, 14, 14), (33, 8, 28, 36), (64, 1, 32, 32), (65, 2, 32, 32), (128, 2, 32, 32),
      (129, 2, 32, 32), (7, 3000, 3, 3), (255, 1, 16, 17)]


@pytest.mark.parametrize("shape", BN, ids=lambda s: "x".join(map(str, s)))
def test_batch_norm(shape):
    rng = np.random.default_rng(sum(shape))
    c = shape[1]
    x, g = (rng.standard_normal(shape) * 1.7 + 40).astype(np.float32), rng.standard_normal(shape).astype(np.float32)
    w, b = rng.standard_normal(c).astype(np.float32), rng.standard_normal(c).astype(np.float32)
    rm, rv = rng.standard_normal(c).astype(np.float32), (rng.random(c) + 0.4).astype(np.float32)
    y, mean, inv, rm_out, rv_out = b200conv.batch_norm_forward(x, w, b, rm, rv, True, 0.23, 1e-4)
    want = bn.forward(x, w, b, rm, rv, True, 0.23, 1e-4, dtype=np.float64)
    assert oracle.rel_l2(y, want[0]) <= 2 * GATE
    for got, e in ((mean, want[1]), (inv, want[2]), (rm_out, want[3]), (rv_out, want[4])):
        np.testing.assert_allclose(got, e, rtol=1e-5, atol=2e-6)
    for got, e in zip(b200conv.batch_norm_backward(g, x, w, mean, inv, True, 1e-4), bn.backward(g, x, w, mean, inv, True, 1e-4, dtype=np.float64)):
        assert oracle.rel_l2(got, e) <= 5 * GATE


# (n, c, h, w), groups
GN = [((1, 2, 1, 1), 2), ((2, 6, 5, 5), 2), ((2, 96, 8, 8), 32), ((1, 40, 40, 40), 2), ((1, 33, 31, 31), 1), ((3, 64, 64, 64), 32), ((1, 64, 32, 32), 1),
      ((1, 65, 32, 32), 1), ((1, 63, 32, 32), 1), ((1, 64, 32, 64), 1), ((1, 64, 33, 64), 1), ((5, 128, 20, 20), 4), ((2, 128, 17, 19), 2)]


@pytest.mark.parametrize("shape,groups", GN, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else f"g{v}")
def test_group_norm(shape, groups):
    rng = np.random.default_rng(sum(shape) + groups)
    x, g = (rng.standard_normal(shape) * 1.5 + 30).astype(np.float32), rng.standard_normal(shape).astype(np.float32)
    w, b = rng.standard_normal(shape[1]).astype(np.float32), rng.standard_normal(shape[1]).astype(np.float32)
    y, mean, rstd = b200conv.group_norm_forward(x, groups, w, b, 1e-5)
    wy, wmean, wrstd = gn.forward(x, groups, w, b, 1e-5, dtype=np.float64)
    if x[0].size > groups:  # one value has nothing to normalise
        assert oracle.rel_l2(y, wy) <= 2 * GATE
    np.testing.assert_allclose(mean, wmean, rtol=2e-6, atol=2e-6)
    np.testing.assert_allclose(rstd, wrstd, rtol=1e-5)
    for got, e in zip(b200conv.group_norm_backward(g, x, mean, rstd, groups, w), gn.backward(g, x, mean, rstd, groups, w, dtype=np.float64)):
        assert np.linalg.norm(got - e) <= 1e-5 * np.linalg.norm(e) + 1e-5 * np.linalg.norm(g) * (x[0].size == groups)


# Training shapes that stream in one direction at least: rows beyond a cluster's registers, and rows that fit but gain nothing by it (norm_plan.cuh), with planes that are
# and are not whole 16-byte pieces, above and below the 256 values at which the streaming arrangement changes
STREAMED_BN = [((40, 70, 61, 61), "rows"), ((66, 200, 33, 33), "rows"), ((70, 560, 17, 17), "rows"), ((460, 500, 7, 7), "cols"), ((600, 70, 16, 16), "rows"), ((1100, 9, 11, 13), "cols")]


@pytest.mark.parametrize("shape,arrangement", STREAMED_BN, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else v)
def test_batch_norm_streamed(shape, arrangement):
    rng = np.random.default_rng(sum(shape))
    c = shape[1]
    x, g = (rng.standard_normal(shape, dtype=np.float32) * np.float32(1.7) + np.float32(4)), rng.standard_normal(shape, dtype=np.float32)
    w, b = rng.standard_normal(c).astype(np.float32), rng.standard_normal(c).astype(np.float32)
    rm, rv = rng.standard_normal(c).astype(np.float32), (rng.random(c) + 0.4).astype(np.float32)
    y, mean, inv, rm_out, rv_out = b200conv.batch_norm_forward(x, w, b, rm, rv, True, 0.23, 1e-4)
    assert b200conv.last_kernel() == f"bn_stats_{arrangement}+finalize+apply"
    want = bn.forward(x, w, b, rm, rv, True, 0.23, 1e-4, dtype=np.float64)
    assert oracle.rel_l2(y, want[0]) <= 2 * GATE
    for got, e in ((mean, want[1]), (inv, want[2]), (rm_out, want[3]), (rv_out, want[4])):
        np.testing.assert_allclose(got, e, rtol=1e-5, atol=2e-6)
    for got, e in zip(b200conv.batch_norm_backward(g, x, w, mean, inv, True, 1e-4), bn.backward(g, x, w, mean, inv, True, 1e-4, dtype=np.float64)):
        assert oracle.rel_l2(got, e) <= 5 * GATE


STREAMED_GN = [((13, 256, 37, 37), 32), ((1, 66, 45, 45), 1), ((3, 40, 63, 65), 1), ((10, 512, 33, 33), 32), ((8, 1152, 33, 33), 32), ((2, 2000, 9, 9), 20)]


@pytest.mark.parametrize("shape,groups", STREAMED_GN, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else f"g{v}")
def test_group_norm_streamed(shape, groups):
    rng = np.random.default_rng(sum(shape) + groups)
    x, g = (rng.standard_normal(shape, dtype=np.float32) * np.float32(1.5) + np.float32(3)), rng.standard_normal(shape, dtype=np.float32)
    w, b = rng.standard_normal(shape[1]).astype(np.float32), rng.standard_normal(shape[1]).astype(np.float32)
    before = b200conv.launch_count()
    y, mean, rstd = b200conv.group_norm_forward(x, groups, w, b, 1e-5)
    assert b200conv.launch_count() == before + 1 and b200conv.last_kernel() == "gn_forward"
    wy, wmean, wrstd = gn.forward(x, groups, w, b, 1e-5, dtype=np.float64)
    assert oracle.rel_l2(y, wy) <= 2 * GATE
    np.testing.assert_allclose(mean, wmean, rtol=2e-6, atol=2e-6)
    np.testing.assert_allclose(rstd, wrstd, rtol=1e-5)
    for got, e in zip(b200conv.group_norm_backward(g, x, mean, rstd, groups, w), gn.backward(g, x, mean, rstd, groups, w, dtype=np.float64)):
        assert oracle.rel_l2(got, e) <= 1e-5


# rank counts between nine and sixteen, one wave of clusters: a share per rank, the last one short
@pytest.mark.parametrize("n,plane", [(73, 32), (107, 32), (127, 32), (37, 33), (45, 31), (37, 32), (61, 32)])
def test_batch_norm_between_nine_and_sixteen_ranks(n, plane):
    rng = np.random.default_rng(n + plane)
    shape, c = (n, 3, plane, plane), 3
    x, g = (rng.standard_normal(shape, dtype=np.float32) + np.float32(2)), rng.standard_normal(shape, dtype=np.float32)
    w, b = rng.standard_normal(c).astype(np.float32), rng.standard_normal(c).astype(np.float32)
    y, mean, inv = b200conv.batch_norm_forward(x, w, b, None, None, True, 0.1, 1e-5)[:3]
    want = bn.forward(x, w, b, None, None, True, 0.1, 1e-5, dtype=np.float64)
    assert oracle.rel_l2(y, want[0]) <= 2 * GATE
    for got, e in zip(b200conv.batch_norm_backward(g, x, w, mean, inv, True, 1e-5), bn.backward(g, x, w, mean, inv, True, 1e-5, dtype=np.float64)):
        assert oracle.rel_l2(got, e) <= 5 * GATE
