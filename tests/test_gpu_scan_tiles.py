"""Scans on both sides of the number of tiles up to which each tile adds up the
ones before it (8,192 of 2,048 elements), through the remesh of a cube whose grid
has a few cells less and a few more, against the host's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [5.0, 26.0, 245.0, 251.0])
def test_remesh_of_large_grids_equals_host(native, scale):
    from visacd_gb300 import build
    build.build_host()
    import visacd_gb300.visacd as V
    V.config.verbose = False
    v = np.array([[x, y, z] for x in (0.0, 1.0) for y in (0.0, 1.0) for z in (0.0, 1.0)])
    t = np.array([[0, 1, 3], [0, 3, 2], [4, 6, 7], [4, 7, 5], [0, 4, 5], [0, 5, 1],
                  [2, 3, 7], [2, 7, 6], [0, 2, 6], [0, 6, 4], [1, 5, 7], [1, 7, 3]], np.int32)
    h = V._manifold_preprocess(v, t, scale, 0.6 / scale)
    g = V._manifold_preprocess_gpu(v, t, scale, 0.6 / scale)
    np.testing.assert_array_equal(g["triangles"], h["triangles"])
    np.testing.assert_array_equal(g["vertices"], h["vertices"])
