"""Visibility at any scale of the coordinates: the edges do not depend on a power of
two, nor does the time (the box test in three products serves meshes up to 1e30),
and a cage much larger or smaller than the part gives the oracle's edges. And the
traversal after a free-space walk is as fast a visit as without one."""
import numpy as np
import pytest

from visacd_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def _f32(m):
    return m[0].astype(np.float32).astype(np.float64), m[1]


def _kernel(ctx, call, reps=6):
    best = 1e9
    for _ in range(reps):
        ctx.set_timing(True)
        try:
            ctx.reset_times()
            call()
            best = min(best, ctx.kernel_times()["visibility"][0])
        finally:
            ctx.set_timing(False)
    return best


@pytest.mark.parametrize("power", [-60, 20, 27, 60, 90])
def test_edges_at_any_scale(ctx, orc, power):
    # (triangle tests ignore hits within 0.001 of the origin: absolute, so the oracle
    # decides at each scale)
    v, t = _f32(mg.displaced_blob(2, seed=3))
    cv, ct = _f32(mg.offset_cage(v, t, 0.03))
    k = 2.0 ** power
    bits, _, _ = orc.visibility(v * k, t, cv * k, ct, use_bvh=False)
    n = len(v)
    sb, cb = ctx.bvh(v * k, t), ctx.bvh(cv * k, ct)
    got, _ = ctx.visibility(v * k, sb, cb)
    have = np.zeros(n * (n - 1) // 2, bool)
    have[orc.linear_from_pairs(got, n)] = True
    bad = (have != (bits & 1).astype(bool)) & ~(bits & 2).astype(bool)
    assert not bad.any(), f"{int(bad.sum())} pairs differ"


@pytest.mark.parametrize("far", [0.0, 1e7, 1e20, 1e29, 1e33])
def test_axis_parallel_segments_beside_a_far_vertex(ctx, orc, far):
    """Segments with components of exactly zero, and a cage or a part with one vertex
    so far out that the least component is no longer 1e-30."""
    g = np.stack(np.meshgrid(*[np.linspace(-1, 1, 6)] * 3, indexing="ij"), -1).reshape(-1, 3)
    cv, ct = _f32(mg.icosphere(2))
    none = np.zeros((0, 3), np.int32)
    n = len(g)
    for which in ("cage", "part"):
        c, p, pt = cv.copy(), g.copy(), none
        if far and which == "cage":
            c = np.concatenate([c, [[far, 0, 0], [far, 1, 0], [far, 0, 1]]])
            ctri = np.concatenate([ct, [[len(cv), len(cv) + 1, len(cv) + 2]]]).astype(np.int32)
        else:
            ctri = ct
        if far and which == "part":
            p = np.concatenate([g, [[far, 0, 0], [far, 1, 0], [far, 0, 1]]])
            pt = np.array([[n, n + 1, n + 2]], np.int32)
        p, c = p.astype(np.float32).astype(np.float64), c.astype(np.float32).astype(np.float64)
        bits, _, _ = orc.visibility(p, pt, c, ctri, use_bvh=False)
        sb, cb = ctx.bvh(p, pt), ctx.bvh(c, ctri)
        got, _ = ctx.visibility(p, sb, cb)
        m = len(p)
        have = np.zeros(m * (m - 1) // 2, bool)
        have[orc.linear_from_pairs(got, m)] = True
        bad = (have != (bits & 1).astype(bool)) & ~(bits & 2).astype(bool)
        assert not bad.any(), f"{which}: {int(bad.sum())} pairs differ"


def test_time_at_large_coordinates(ctx):
    """A blob of 2,562 vertices at 1e8: the time of the same at 1 (1.25 times before
    the box test served it)."""
    def call(k):
        v, t = mg.displaced_blob(4, seed=3)
        cage = mg.offset_cage(v, t, 0.03)
        sb, cb = ctx.bvh(v * k, t), ctx.bvh(cage[0] * k, cage[1])
        return lambda: ctx.visibility(v * k, sb, cb)

    assert _kernel(ctx, call(1e8)) <= 1.12 * _kernel(ctx, call(1.0))


def test_time_after_a_walk(ctx):
    """18 million pairs of random points, of which the walk clears an eighth of the
    visits: the traversal takes 0.93 of its time without a walk (1.005 when its copy
    for listed tiles spilled)."""
    p = np.random.default_rng(6000).uniform(-1, 1, (6000, 3)).astype(np.float32)
    sb, cb = ctx.bvh(p, np.zeros((0, 3), np.int32)), ctx.bvh(*mg.icosphere(4))
    after = _kernel(ctx, lambda: ctx.visibility(p, sb, cb))
    ctx.set_vis_trace(False)
    try:
        alone = _kernel(ctx, lambda: ctx.visibility(p, sb, cb))
    finally:
        ctx.set_vis_trace(True)
    assert after <= 0.97 * alone
