"""Gradients of the proposer's per-edge layers, which run over the rows that the
max-pool selects: few and many selected rows, equal rows (ties go to the first),
channels that pool to zero, odd batches. Against the BF16-emulating oracle, with
the tolerance of the gradient test of the whole batch (BF16 operands, FP32 sums
in another order)."""
import numpy as np
import pytest

import test_gpu_learned as tl

pytestmark = pytest.mark.gpu
lr = tl.lr


@pytest.mark.parametrize("B", [1, 2, 5, 17])
@pytest.mark.parametrize("rows", ["all", "three", "one", "dead"])
def test_gradients_over_selected_rows(native, ctx, B, rows):
    params = lr.init_params(9)
    feats, labels, w = tl._case(21 + B, B=B)
    feats = feats.copy()
    if rows == "three":  # the same three rows over and over
        feats = np.ascontiguousarray(feats[:, np.arange(feats.shape[1]) % 3])
    if rows == "one":
        feats = np.ascontiguousarray(np.repeat(feats[:, :1], feats.shape[1], axis=1))
    if rows == "dead":  # half of the pooled channels never positive
        params = params.copy()
        params[lr.BOFF[2]:lr.BOFF[2] + 128] = -100.0
    lp = native.PlaneProposer(ctx, params=params)
    loss, g = lp.grads(feats, labels, w)
    rloss, rg, _ = lr.forward_backward(params, feats, labels, w, emulate_bf16=True)
    assert abs(loss - rloss) <= 1e-3 * abs(rloss)
    for l in range(6):
        for lo, n in ((lr.WOFF[l], lr.K[l] * lr.N[l]), (lr.BOFF[l], lr.N[l])):
            a, b = g[lo:lo + n], rg[lo:lo + n]
            assert np.linalg.norm(a - b) <= tl.GRAD_RTOL * max(np.linalg.norm(b), 1e-30), (l, n)
