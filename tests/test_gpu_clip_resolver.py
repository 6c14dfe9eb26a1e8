"""The clip's border resolver at the sizes and inputs where its two forms meet:
all touching triangles at once (up to 2048), and the ordered walk beyond that,
for planes through vertices and for very many coincident border points. Both
must give the host clip's parts, maps and border, bit for bit."""
import numpy as np
import pytest

from visacd_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def V():
    from visacd_gb300 import build
    build.build_host()
    from visacd_gb300 import visacd
    return visacd


def _unit(x):
    return [float(c) for c in np.asarray(x, dtype=np.float64) / np.linalg.norm(x)]


CASES = {
    # touching triangles: few, around a warp, around the block, at the limit, beyond it
    "tetrahedron": (lambda: mg.icosphere(0), _unit([0.31, 0.42, 0.85]) + [0.1]),
    "icosphere2": (lambda: mg.displaced_blob(2, seed=3), _unit([0.3, -0.2, 0.9]) + [0.05]),
    "torus_514_touching": (lambda: mg.torus(nu=128, nv=5, seed=1), _unit([0.01, 0.02, 1.0]) + [0.003]),
    "torus_2044_touching": (lambda: mg.torus(nu=511, nv=6, seed=2), _unit([0.0, 0.0, 1.0]) + [0.1]),
    "torus_2052_touching": (lambda: mg.torus(nu=513, nv=6, seed=2), _unit([0.0, 0.0, 1.0]) + [0.1]),
    "torus_4400_touching": (lambda: mg.torus(nu=1100, nv=6, seed=4), _unit([0.0, 0.0, 1.0]) + [0.1]),
    # the plane through vertices of crossed triangles (unperturbed rings)
    "torus_vertices": (lambda: mg.torus(nu=40, nv=8, perturb=0.0), [1.0, 0.0, 0.0, 0.0]),
    "torus_vertices_large": (lambda: mg.torus(nu=1200, nv=4, perturb=0.0), [0.0, 0.0, 1.0, 0.0]),
    "icosphere4_axis": (lambda: mg.icosphere(4), [0.0, 1.0, 0.0, 0.0]),
    # points closer than the 1e-4 merge distance: some, chains, nearly all
    "small_1e-2": (lambda: _scaled(mg.displaced_blob(4, seed=5), 1e-2), _unit([0.2, 0.5, 0.7]) + [0.0]),
    "small_2e-3": (lambda: _scaled(mg.displaced_blob(4, seed=6), 2e-3), _unit([0.2, 0.5, 0.7]) + [0.0]),
    "small_2e-4": (lambda: _scaled(mg.displaced_blob(4, seed=7), 2e-4), _unit([0.2, 0.5, 0.7]) + [0.0]),
    "far_from_origin": (lambda: _moved(mg.displaced_blob(3, seed=8), 300.0), _unit([0.1, 0.9, 0.3]) + [-408.8]),
}


def _scaled(m, k):
    return m[0] * k, m[1]


def _moved(m, d):
    return m[0] + d, m[1]


@pytest.mark.parametrize("name", CASES)
def test_resolver_equals_host(V, ctx, name):
    make, plane = CASES[name]
    v, t = make()
    a, am1, am2 = V._clip(v, t, plane)
    b, bm1, bm2 = V._clip_gpu(v, t, plane)
    np.testing.assert_array_equal(am1, bm1)
    np.testing.assert_array_equal(am2, bm2)
    assert len(a) == len(b)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x["vertices"], y["vertices"])
        np.testing.assert_array_equal(x["triangles"], y["triangles"])
        np.testing.assert_array_equal(x["is_new"], y["is_new"])
    if "touching" in name:
        assert ctx.clip(v, t, plane)["n_touching"] == int(name.split("_")[1])


def test_resolver_on_clipped_parts(V):
    # halves of halves: caps, slivers and the coincidences along earlier cuts
    rng = np.random.default_rng(11)
    v, t = mg.displaced_blob(4, seed=12)
    parts = [(v, t)]
    for _ in range(4):
        nxt = []
        for v, t in parts:
            n = rng.normal(size=3)
            n /= np.linalg.norm(n)
            pl = [*n, -float(n @ v.mean(axis=0))]
            a, am1, am2 = V._clip(v, t, pl)
            b, bm1, bm2 = V._clip_gpu(v, t, pl)
            np.testing.assert_array_equal(am1, bm1)
            np.testing.assert_array_equal(am2, bm2)
            assert len(a) == len(b)
            for x, y in zip(a, b):
                np.testing.assert_array_equal(x["vertices"], y["vertices"])
                np.testing.assert_array_equal(x["triangles"], y["triangles"])
            nxt += [(h["vertices"], h["triangles"]) for h in a]
        parts = nxt
