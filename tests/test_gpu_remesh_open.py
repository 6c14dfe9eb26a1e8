"""Remeshing of open meshes, whose votes change across the opening, far from any
triangle: the mesh is the host restatement's bit for bit, and large triangles are
shared out over the GPU in the pass that serves those voxels too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(faces):
    v = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], float)
    q = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)][:faces]
    return v, np.array([t for a, b, c, d in q for t in ((a, b, c), (a, c, d))], np.int32)


def _bowl_in_a_box():
    """Two large faces beside the small triangles of a bowl."""
    from visacd_gb300 import meshgen as mg
    v, t = mg.icosphere(4)
    t = t[v[t].mean(1)[:, 2] < 0.3]
    b, f = _box(4)
    return np.concatenate([0.8 * v, b]), np.concatenate([t, f + len(v)]).astype(np.int32)


@pytest.mark.parametrize("scale", [3.0, 11.0, 40.0])
@pytest.mark.parametrize("kind", ["open box", "two faces", "bowl in a box"])
@pytest.mark.parametrize("iso", [0.05, 0.7, 2.0])
def test_open_meshes_equal_host(native, kind, scale, iso):
    from visacd_gb300 import build
    build.build_host()
    import visacd_gb300.visacd as V
    v, t = {"open box": lambda: _box(5), "two faces": lambda: _box(2), "bowl in a box": _bowl_in_a_box}[kind]()
    h = V._manifold_preprocess(v, t, scale, iso / scale)
    g = V._manifold_preprocess_gpu(v, t, scale, iso / scale)
    np.testing.assert_array_equal(g["triangles"], h["triangles"])
    np.testing.assert_array_equal(g["vertices"], h["vertices"])


def test_large_faces_are_shared_out(ctx):
    """Ten faces of 200 x 200 voxels: distance kernels of the open box against the
    closed one's (which has no voxels for the second pass), the least of six calls:
    8 times as long when a face of that pass is one warp's."""
    def kernels(faces):
        best = 1e9
        for _ in range(6):
            ctx.set_timing(True)
            try:
                ctx.reset_times()
                ctx.sdf_remesh(*_box(faces), 100.0, 0.05)
                best = min(best, ctx.kernel_times()["sdf_dist"][0])
            finally:
                ctx.set_timing(False)
        return best

    assert kernels(5) <= 3 * kernels(6)
