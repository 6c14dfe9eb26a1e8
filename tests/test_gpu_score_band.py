"""Scoring by vertex sides where most of a block's values lie in their rounding band:
512 vertices 1e-6 above or below a plane against 32 copies of it moved by a few
roundings, more than 8,192 values that need FP64 in one block of 512 vertices and 32
planes, whose list holds 2,048. Other planes and vertices stand beside them. The
scores are the FP64 oracle's integers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [512, 700, 1024])
@pytest.mark.parametrize("P", [32, 45])
def test_block_of_band_values(ctx, orc, N, P):
    rng = np.random.default_rng(N + P)
    n = np.array([1.0, 2.0, 3.0])
    n = (n / np.linalg.norm(n)).astype(np.float32).astype(np.float64)
    v = rng.uniform(-1, 1, (N, 3))
    v[:512] -= np.outer(v[:512] @ n - rng.choice([-1e-6, 1e-6], 512), n) / (n @ n)
    v = v.astype(np.float32)
    planes = np.zeros((P, 4), np.float32)
    planes[:, :3] = n
    planes[:, 3] = rng.integers(-2, 3, P) * 3e-8
    planes[32:] = rng.normal(size=(P - 32, 4))
    # Within 1.2e-7 S of +-1e-6, S = |n_x| max|x| + |n_y| max|y| + |n_z| max|z|, a value is
    # in the band (3e-7 S to both sides) after its FP32 roundings (1.8e-7 S) too.
    value = np.abs((v[:512].astype(np.float64) @ n)[:, None] + planes[:32, 3].astype(np.float64))
    assert (np.abs(value - 1e-6) < 1.2e-7 * (np.abs(n) @ np.abs(v).max(0))).sum() > 4 * 2048
    assert (value > 1e-6).mean() > 0.1 and (value < 1e-6).mean() > 0.1
    e = rng.integers(0, N, (N + 5000, 2)).astype(np.uint32)
    got, st = ctx.score_planes(planes, v, e)
    _, q, qexp, _ = orc.score_planes(planes, v, e)
    assert (q[:32] > 0).any()
    np.testing.assert_array_equal(got, np.ldexp(q.astype(np.float64), qexp))
    assert st["argmax"] == int(np.argmax(got))
