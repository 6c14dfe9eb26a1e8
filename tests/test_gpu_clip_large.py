"""Cuts of large meshes that few triangles touch: the ordered walk of the border
resolver gives the host's parts, and takes the time its touching triangles need,
however many others there are."""
import numpy as np
import pytest

from visacd_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def _with_far_triangles(m, n):
    """m beside a fine sphere far above it."""
    v, t = m
    s, f = mg.icosphere(n)
    return np.concatenate([v, s + [0, 0, 9.0]]), np.concatenate([t, f + len(v)]).astype(np.int32)


CASES = {
    "through vertices": (lambda: mg.torus(nu=1200, nv=4, perturb=0.0), [0.0, 0.0, 1.0, 0.0]),
    "beyond the parallel form": (lambda: mg.torus(nu=513, nv=6, seed=2), [0.0, 0.0, 1.0, 0.1]),
    "few through vertices": (lambda: mg.torus(nu=40, nv=8, perturb=0.0), [0.0, 0.0, 1.0, 0.0]),
}


@pytest.mark.parametrize("name", CASES)
def test_ordered_walk_beside_many_triangles(ctx, native, name):
    from visacd_gb300 import build
    build.build_host()
    from visacd_gb300 import visacd as V
    make, plane = CASES[name]
    v, t = _with_far_triangles(make(), 5)
    a, am1, am2 = V._clip(v, t, plane)
    b, bm1, bm2 = V._clip_gpu(v, t, plane)
    np.testing.assert_array_equal(am1, bm1)
    np.testing.assert_array_equal(am2, bm2)
    assert len(a) == len(b)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x["vertices"], y["vertices"])
        np.testing.assert_array_equal(x["triangles"], y["triangles"])


def test_resolver_time_follows_the_touching_triangles(ctx):
    """Kernel time of the resolver with 1.3 million triangles more, the least of four
    calls: they are looked through (0.3 ms), and took 13 ms more when tables of their
    size were emptied."""
    def resolve(mesh, plane):
        best = 1e9
        for _ in range(4):
            ctx.set_timing(True)
            try:
                ctx.reset_times()
                ctx.clip(*mesh, plane)
                best = min(best, ctx.kernel_times()["clip_resolve"][0])
            finally:
                ctx.set_timing(False)
        return best

    make, plane = CASES["through vertices"]
    assert resolve(_with_far_triangles(make(), 8), plane) <= 1.2 * resolve(make(), plane) + 1.0
