"""Which voxels of the GPU remesh get an exact distance: levels on both sides of
one voxel (and at or below zero), open meshes whose votes differ without a
surface between, triangles covering many rays, grids of odd extents. The mesh
equals the host restatement bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def V(native):
    from visacd_gb300 import build
    build.build_host()
    import visacd_gb300.visacd as V
    V.config.verbose = False
    return V


def _mesh(kind):
    from visacd_gb300 import meshgen as mg
    if kind == "cube":  # two triangles per face: every ray box is wide
        return _cube()
    v, t = mg.displaced_blob(3, seed=4)
    v = v / np.abs(v).max()
    if kind == "open":  # a third of the triangles gone
        return v, np.ascontiguousarray(t[np.arange(len(t)) % 3 != 0])
    if kind == "half":  # one side gone, so whole rays cross once
        return v, np.ascontiguousarray(t[v[t].mean(1)[:, 0] < 0.2])
    return v * [1.0, 0.37, 0.71], t


def _cube():
    v = np.array([[x, y, z] for x in (-.5, .5) for y in (-.5, .5) for z in (-.5, .5)], float)
    t = np.array([[0, 1, 3], [0, 3, 2], [4, 6, 7], [4, 7, 5], [0, 4, 5], [0, 5, 1],
                  [2, 3, 7], [2, 7, 6], [0, 2, 6], [0, 6, 4], [1, 5, 7], [1, 7, 3]], np.int32)
    return v, t


@pytest.mark.parametrize("kind", ["cube", "open", "half", "flat"])
@pytest.mark.parametrize("scale", [7.0, 23.0])
@pytest.mark.parametrize("iso", [-0.5, 0.0, 0.05, 0.55, 1.0, 1.2, 3.5])
def test_field_ranges_equal_host(V, kind, scale, iso):
    v, t = _mesh(kind)
    h = V._manifold_preprocess(v, t, scale, iso / scale)
    g = V._manifold_preprocess_gpu(v, t, scale, iso / scale)
    np.testing.assert_array_equal(g["triangles"], h["triangles"])
    np.testing.assert_array_equal(g["vertices"], h["vertices"])
