"""BVH builds and point orders at the sizes where the one-launch build changes
shape: one triangle, runs of 32 and groups of 1024 leaves, the switch from one
CTA to a cluster (2048) and to the general build (131072). A wrong box, split or
order loses hits, so visibility over the mesh is compared with the FP64 oracle;
the depth is checked against the tree's possible range."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(nt: int, seed: int):
    """nt small triangles scattered over the shell between two cubes, a tenth of
    them repeated (equal Morton codes)."""
    rng = np.random.default_rng([seed, nt])
    c = rng.uniform(-1, 1, size=(nt, 3))
    c /= np.maximum(np.abs(c).max(axis=1, keepdims=True), 1e-3)
    c *= rng.uniform(0.6, 0.9, size=(nt, 1))
    c[rng.random(nt) < 0.1] = c[0]
    size = 1.5 / math.sqrt(max(nt, 4))
    v = c[:, None, :] + rng.normal(scale=size, size=(nt, 3, 3))
    return v.reshape(-1, 3).astype(np.float32).astype(np.float64), np.arange(3 * nt, dtype=np.int32).reshape(-1, 3)


def _compare(ctx, orc, pts, cage, mask=None):
    none = np.zeros((0, 3), np.int32)
    sb, cb = ctx.bvh(pts, none), ctx.bvh(*cage)
    got, _ = ctx.visibility(pts, sb, cb, is_new=mask)
    bits, _, _ = orc.visibility(pts, none, *cage, use_bvh=False)
    n = len(pts)
    have = np.zeros(n * (n - 1) // 2, bool)
    have[orc.linear_from_pairs(got, n)] = True
    want, graze = (bits & 1).astype(bool), (bits & 2).astype(bool)
    if mask is not None:
        i, j = np.triu_indices(n, 1)
        want &= (mask[i] | mask[j]).astype(bool)
    bad = (have != want) & ~graze
    assert not bad.any(), f"{int(bad.sum())} pairs differ"
    depth = cb.info()[1]
    sb.close()
    cb.close()
    return depth, int(want.sum())


@pytest.mark.parametrize("nt", [1, 2, 3, 31, 32, 33, 63, 64, 65, 1023, 1024, 1025, 1056, 2047, 2048, 2049, 2080, 4097,
                                32767, 32769, 33 * 1024 + 7, 65536, 131071, 131072, 131073])
def test_build_sizes(ctx, orc, nt):
    rng = np.random.default_rng(nt)
    pts = rng.uniform(-1, 1, size=(24, 3)).astype(np.float32).astype(np.float64)
    depth, hits = _compare(ctx, orc, pts, _soup(nt, 1))
    assert math.ceil(math.log2(max(nt, 2))) <= depth <= max(nt - 1, 1)
    assert nt < 64 or hits > 0


@pytest.mark.parametrize("n", [2, 3, 31, 33, 255, 257, 1000])
def test_point_order_masked(ctx, orc, n):
    rng = np.random.default_rng(n)
    pts = rng.uniform(-1, 1, size=(n, 3)).astype(np.float32).astype(np.float64)
    for frac in (0.0, 0.1, 1.0):
        _compare(ctx, orc, pts, _soup(200, 2), mask=(rng.random(n) < frac).astype(np.uint8))


def test_point_order_cluster(ctx):
    """Point sets on both sides of the cluster switch and of the general sort,
    masked and not: the masked call's pairs are the unmasked call's with a new
    endpoint."""
    cage = _soup(500, 3)
    none = np.zeros((0, 3), np.int32)
    for n in (2048, 2049, 5003):
        rng = np.random.default_rng(n)
        pts = rng.uniform(-1, 1, size=(n, 3)).astype(np.float32)
        mask = (rng.random(n) < 0.05).astype(np.uint8)
        sb, cb = ctx.bvh(pts, none), ctx.bvh(*cage)
        full, st = ctx.visibility(pts, sb, cb)
        part, sm = ctx.visibility(pts, sb, cb, is_new=mask)
        keep = (mask[full[:, 0]] | mask[full[:, 1]]).astype(bool)
        np.testing.assert_array_equal(part, full[keep])
        old = int((mask == 0).sum())
        assert st["pairs_tested"] == n * (n - 1) // 2
        assert sm["pairs_tested"] == n * (n - 1) // 2 - old * (old - 1) // 2
        both, sb2 = ctx.visibility_batch([(pts, sb, cb, None), (pts, sb, cb, mask)])
        np.testing.assert_array_equal(both[0], full)
        np.testing.assert_array_equal(both[1], part)
        sb.close()
        cb.close()


def test_large_masked_points(ctx):
    """Above 131072 points the general sort orders them (one new point)."""
    n = 131073
    rng = np.random.default_rng(5)
    pts = rng.uniform(-1, 1, size=(n, 3)).astype(np.float32)
    mask = np.zeros(n, np.uint8)
    mask[777] = 1
    cage = _soup(60, 4)
    none = np.zeros((0, 3), np.int32)
    sb, cb = ctx.bvh(pts, none), ctx.bvh(*cage)
    e, st = ctx.visibility(pts, sb, cb, is_new=mask)
    assert st["pairs_tested"] == n - 1 and len(e) == st["n_edges"]
    assert (e == 777).any(axis=1).all()
    # the same pairs in a small call: the new point with every 97th other
    idx = np.concatenate([[777], np.setdiff1d(np.arange(0, n, 97), [777])])
    sub, _ = ctx.visibility(pts[idx], ctx.bvh(pts[idx], none), cb)
    other = set(int(x) for x in e[(e[:, 0] == 777) | (e[:, 1] == 777)].sum(axis=1) - 777)
    small = set(int(idx[j]) for i, j in sub if i == 0)
    assert small == other & set(int(x) for x in idx[1:])


def test_build_is_seen_by_another_context(native, ctx):
    """A BVH built on one context and used at once on another."""
    cage = _soup(60000, 6)
    rng = np.random.default_rng(8)
    pts = rng.uniform(-1, 1, size=(300, 3)).astype(np.float32)
    none = np.zeros((0, 3), np.int32)
    other = native.Context(0)
    for _ in range(3):
        sb, cb = other.bvh(pts, none), other.bvh(*cage)
        a, _ = ctx.visibility(pts, sb, cb)
        b, _ = other.visibility(pts, sb, cb)
        np.testing.assert_array_equal(a, b)
        sb.close()
        cb.close()
    other.close()


def test_bad_index_is_refused(native, ctx):
    v, t = _soup(50, 7)
    t = t.copy()
    t[17, 2] = len(v)
    with pytest.raises(native.VisacdError):
        ctx.bvh(v, t)
