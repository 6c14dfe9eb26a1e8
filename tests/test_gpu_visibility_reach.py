"""Visibility calls large enough for the free-space walk and its table of free
reaches by direction: the edges equal those of the traversal alone (the walk
switched off), for whole, masked and batched calls, with full tables, small
ones (few new points among many) and none, on bodies where segments run inside,
outside and through the cage."""
import numpy as np
import pytest

from visacd_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def _body(kind, level=4):
    if kind == "torus":
        v, t = mg.torus(nu=90, nv=40, seed=3)
    elif kind == "box":  # axis-parallel segments, ties between the largest components
        v, t = mg.icosphere(level)
        v = np.clip(v, -0.6, 0.6)
    else:
        v, t = mg.displaced_blob(level, seed=6)
    return v, t


def _parts(kind):
    v, t = _body(kind, 4)
    n = mg.vertex_normals(v, t)
    # more points than vertices: on the surface, slightly inside and outside the cage
    rng = np.random.default_rng(1)
    k = rng.integers(len(v), size=3200 - len(v) if len(v) < 3200 else 0)
    far = np.concatenate([v, v[k] + n[k] * rng.uniform(-0.3, 0.08, (len(k), 1))])
    return far, v, t, *mg.offset_cage(v, t, 0.03)


def _edges(ctx, parts, on):
    ctx.set_vis_trace(on)
    try:
        return ctx.visibility_batch(parts)[0]
    finally:
        ctx.set_vis_trace(True)


@pytest.mark.parametrize("kind", ["blob", "torus", "box"])
@pytest.mark.parametrize("masked", [False, True])
def test_walk_equals_traversal(ctx, kind, masked):
    p, v, t, cv, ct = _parts(kind)
    p = np.ascontiguousarray(p, np.float32)
    new = None
    if masked:
        new = np.zeros(len(p), np.uint8)
        new[::2] = 1
    a, b = ctx.bvh(p, t), ctx.bvh(cv, ct)  # (the points are the vertices; some in no triangle)
    small = _body("blob", 2)
    sa, sb = ctx.bvh(*small), ctx.bvh(*mg.offset_cage(*small, 0.03))
    parts = [(small[0], sa, sb, None), (p, a, b, new), (small[0], sa, sb, None), (p, a, b, None)]
    for got, want in zip(_edges(ctx, parts, True), _edges(ctx, parts, False)):
        assert len(want) > 0
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("n,n_new", [(6000, 900), (20000, 260), (60000, 75), (3000, 3000)])
def test_walk_with_few_new_points(ctx, n, n_new):
    v, t = _body("blob", 4)
    rng = np.random.default_rng(n)
    k = rng.integers(len(v), size=n - len(v))
    p = np.concatenate([v, v[k] * rng.uniform(0.9, 1.0, (len(k), 1))])
    new = np.zeros(n, np.uint8)
    new[rng.permutation(n)[:n_new]] = 1
    parts = [(p, ctx.bvh(p, t), ctx.bvh(*mg.offset_cage(v, t, 0.03)), new)]
    np.testing.assert_array_equal(_edges(ctx, parts, True)[0], _edges(ctx, parts, False)[0])
