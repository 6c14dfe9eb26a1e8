"""Candidate planes of vertices far from the origin: plane offsets of some
thousands, whose FP32 rounding is a good part of the 1e-3 within which two planes
are similar. The planes are the oracle's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0.0, 20.0, 1000.0, 30000.0])
def test_similar_planes_far_from_the_origin(ctx, orc, shift):
    rng = np.random.default_rng(4)
    n = 400
    v = np.stack([rng.uniform(0, 0.5, n), np.zeros(n), np.zeros(n)], 1) + shift  # all edges along x
    i, j = rng.integers(0, n, 8000), rng.integers(0, n, 8000)
    e = np.stack([np.minimum(i, j), np.maximum(i, j)], 1)[i != j].astype(np.uint32)
    want, draws, used = orc.candidate_planes_with_draws(v, e, 4000, 9)
    got, got_used = ctx.candidate_planes(v, e, draws, 4000)
    assert 0 < len(want) < len(np.unique(draws))  # many dropped as similar
    np.testing.assert_array_equal(got, want)
    assert got_used == used
