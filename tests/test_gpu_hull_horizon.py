"""Hull steps that replace many faces at once (visacd_convex_hulls): rings whose
horizon passes 32 edges, whose new faces pass 64 and whose flood fill goes more
than 8 deep, against the host QuickHull, triangle for triangle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rings():
    """A ring seen from a point on either side of it; its own heights decide in
    which order its faces appear."""
    for n in (31, 32, 33, 34, 63, 64, 65, 66, 400, 1500):
        for noise in (1e-9, 1e-5, 1e-3):
            rng = np.random.default_rng(n)
            for even in (False, True):
                a = np.arange(n) * 2 * np.pi / n if even else rng.uniform(0, 2 * np.pi, n)
                yield np.r_[np.c_[np.cos(a), np.sin(a), rng.normal(scale=noise, size=n)],
                            [[0, 0, 0.0025]], [[0.1, 0.1, -2.0]]]
    a = np.arange(400) * 2 * np.pi / 400  # 14 deep
    z = np.random.default_rng(504958321).normal(scale=1.1405181306036275e-05, size=400)
    yield np.r_[np.c_[np.cos(a), np.sin(a), z], [[0, 0, 0.2092598184224765]], [[0.1, 0.1, -2.0]]]


@pytest.mark.parametrize("fix", [True, False])
def test_gpu_hull_large_horizons_equal_host(native, ctx, fix):
    from visacd_gb300 import build
    build.build_host()
    import visacd_gb300.visacd as V
    sets = list(rings())
    for p, g in zip(sets, ctx.convex_hulls(sets, fix_normals=fix)):
        want = np.asarray(V._convex_hull(p, fix)["triangles"], np.int32).reshape(-1, 3)
        assert np.array_equal(g, want), len(p)
