"""Meshes and points with infinite coordinates: the boxes around such a vertex are
infinite, and neither box test may lose the finite triangles below them. The
edges are the FP64 oracle's (every triangle tested)."""
import numpy as np
import pytest

from visacd_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [1.0, 8.0])  # points within the cage's scale, and beyond four times it
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("where", ["part", "cage", "both", "cage, two ways"])
def test_infinite_vertices(ctx, orc, where, value, far):
    v, t = mg.displaced_blob(3, seed=3)
    cv, ct = mg.offset_cage(v, t, 0.03)
    v, cv = (v * far).astype(np.float32).astype(np.float64), cv.astype(np.float32).astype(np.float64)
    if where in ("part", "both"):
        v[5, 1] = value
    if where != "part":
        cv[5, 1] = value
    if where == "cage, two ways":  # neighbours, one at each end
        cv[ct[(ct == 5).any(axis=1)][0]] = [[0.0, value, 0.0], [0.0, -value, 0.1], [0.3, value, 0.0]]
    bits, _, _ = orc.visibility(v, t, cv, ct, use_bvh=False)
    n = len(v)
    want, graze = (bits & 1).astype(bool), (bits & 2).astype(bool)
    sb, cb = ctx.bvh(v, t), ctx.bvh(cv, ct)
    got, _ = ctx.visibility(v, sb, cb)
    together, _ = ctx.compute_intersection_matrix(v, t, cv, ct)
    for e in (got, together):
        have = np.zeros(n * (n - 1) // 2, bool)
        have[orc.linear_from_pairs(e, n)] = True
        bad = (have != want) & ~graze
        assert not bad.any(), f"{int(bad.sum())} pairs differ"
    sb.close()
    cb.close()
