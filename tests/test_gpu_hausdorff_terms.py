"""Sampled face Hausdorff distances (visacd_face_hausdorff_batch) against exact
nearest samples and true triangle distances in FP64: queries far from the other
surface (many rings of cells), fewer than 10 samples, lists of one and of
several queries per warp, and repeated samples (equal distances at the tenth
place). The triangles are regular, where the metric's formula is the true
distance; both sides round a few hundred FP64 operations on values of order 1,
so they agree to 1e-11."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _surface(n, seed, shift=(0.0, 0.0, 0.0), scale=1.0, repeat=1):
    from visacd_gb300 import meshgen as mg
    v, t = mg.icosphere(3)
    v = v * scale + np.asarray(shift)
    rng = np.random.default_rng(seed)
    ids = rng.integers(len(t), size=n)
    b = rng.dirichlet([1, 1, 1], size=n)
    x = (v[t[ids]] * b[:, :, None]).sum(1)
    return v, t.astype(np.int32), np.repeat(x, repeat, 0), np.repeat(ids, repeat).astype(np.int32)


def _tri_dist(p, a, b, c):
    """Distance of points to triangles, row by row: the plane distance where the
    projection falls inside, else the least distance to the three segments."""
    n = np.cross(b - a, c - a)
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    h = ((p - a) * n).sum(1)
    inside = np.ones(len(p), bool)
    best = np.full(len(p), np.inf)
    for s, e in ((a, b), (b, c), (c, a)):
        inside &= (np.cross(e - s, p - s) * n).sum(1) >= 0
        u = np.clip(((p - s) * (e - s)).sum(1) / ((e - s) ** 2).sum(1), 0, 1)
        best = np.minimum(best, np.linalg.norm(p - s - u[:, None] * (e - s), axis=1))
    return np.where(inside, np.abs(h), best)


def _directed(xq, v, t, x, ids):
    tree = pytest.importorskip("scipy.spatial").cKDTree(x)
    k = min(10, len(x))
    near = tree.query(xq, k=k)[1].reshape(len(xq), k)
    tri = t[ids[near]].reshape(-1, 3)
    d = _tri_dist(np.repeat(xq, k, 0), v[tri[:, 0]], v[tri[:, 1]], v[tri[:, 2]]).reshape(-1, k)
    return d.min(1).max()


@pytest.mark.parametrize("pair", [
    (dict(n=1, seed=1), dict(n=1, seed=2)),
    (dict(n=9, seed=1), dict(n=11, seed=2, shift=(0.1, 0, 0))),
    (dict(n=33, seed=1), dict(n=4000, seed=2, shift=(3.0, 1.0, 0))),
    (dict(n=4000, seed=1), dict(n=4000, seed=2, scale=0.4, shift=(0.2, 0, 0))),
    (dict(n=20000, seed=1), dict(n=20000, seed=2)),
    (dict(n=30000, seed=1), dict(n=25000, seed=2, scale=1.03)),
    (dict(n=700, seed=1, repeat=12), dict(n=900, seed=2, scale=0.9, repeat=11)),
])
@pytest.mark.parametrize("independent", [True, False])
def test_terms_equal_exact_neighbours(ctx, pair, independent):
    a, b = _surface(**pair[0]), _surface(**pair[1])
    want = max(_directed(a[2], b[0], b[1], b[2], b[3]), _directed(b[2], a[0], a[1], a[2], a[3]))
    other = _surface(500, 7), _surface(400, 8, scale=0.99)
    low = max(_directed(other[0][2], *other[1]), _directed(other[1][2], *other[0]))
    got = ctx.face_hausdorff_batch([a + b, other[0] + other[1]], independent=independent)
    if independent or want >= low:
        assert abs(got[0] - want) <= 1e-11
    if independent or low >= want:
        assert abs(got[1] - low) <= 1e-11
