"""Scoring by vertex sides (calls with no fewer edges than vertices and at most
24,576 vertices): on both sides of its limits and at the remainders of 32 planes,
32 edges and 512 vertices the scores are those of the per-edge kernel (a forced
number of planes per thread) and the FP64 oracle's integers, with vertices on and
within rounding of a plane's +-1e-6, skipped edges, NaN planes and planes whose
FP32 bound overflows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,E,P", [(1, 1, 1), (2, 4, 31), (3, 3, 32), (31, 30, 33), (511, 511, 64), (512, 1024, 65),
                                   (513, 30000, 97), (642, 4661, 592), (2562, 59183, 129), (24576, 24576, 40),
                                   (24576, 24575, 40), (24577, 49200, 40)])
def test_sides_equal_the_per_edge_kernel(ctx, orc, N, E, P):
    rng = np.random.default_rng(N * 31 + E + P)
    v = rng.normal(size=(N, 3)).astype(np.float32)
    n = rng.normal(size=(P, 3))
    planes = np.c_[n / np.linalg.norm(n, axis=1, keepdims=True), rng.uniform(-0.5, 0.5, P)].astype(np.float32)
    planes[::3, 3] = -(planes[::3, :3].astype(np.float64) * v[rng.integers(0, N, len(planes[::3]))]).sum(1)
    # A third of the vertices within a few roundings of plane 0's +-1e-6.
    near = np.arange(0, N, 3)
    d = v[near].astype(np.float64) @ planes[0, :3].astype(np.float64) + planes[0, 3]
    off = rng.choice([-1.0, 1.0], len(near)) * (1e-6 + rng.integers(-3, 4, len(near)) * 6e-8)
    v[near] = (v[near] - (d - off)[:, None] * planes[0, :3].astype(np.float64)).astype(np.float32)
    e = rng.integers(0, N, (E, 2)).astype(np.uint32)
    e[::17, 0] = N + 5
    if N > 100:
        v[7], v[8, 1] = np.nan, np.inf
    if P > 40:
        planes[37] = np.nan
    ctx.set_score_k(0)
    got, st = ctx.score_planes(planes, v, e)
    try:
        ctx.set_score_k(1)
        want, st1 = ctx.score_planes(planes, v, e)
    finally:
        ctx.set_score_k(0)
    np.testing.assert_array_equal(got, want)
    assert st["argmax"] == st1["argmax"] and st["skipped_edges"] == st1["skipped_edges"]
    _, q, qexp, _ = orc.score_planes(planes, v, e)
    np.testing.assert_array_equal(got, np.ldexp(q.astype(np.float64), qexp))
    big = planes.copy()
    big[:, :] *= np.float32(1e38)
    _, q, qexp, _ = orc.score_planes(big, v, e)
    np.testing.assert_array_equal(ctx.score_planes(big, v, e)[0], np.ldexp(q.astype(np.float64), qexp))
