"""Remeshing of meshes with degenerate triangles (repeated vertices, collinear or
nearly collinear corners, points): where the distance formula gives a wrong value or
NaN on them the host uses or ignores it, and the GPU has to do the same. The mesh
equals the host restatement's bit for bit."""
import numpy as np
import pytest

from visacd_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def _mesh(kind, rng):
    v, t = mg.displaced_blob(2, seed=int(rng.integers(1000)))
    if kind == "integers":
        n = int(rng.integers(4, 40))
        return rng.integers(-2, 3, (n, 3)).astype(float), rng.integers(0, n, (int(rng.integers(4, 60)), 3))
    if kind == "rounded":
        return np.round(v * 4) / 4, t
    if kind == "repeated":
        extra = rng.integers(0, len(v), (20, 3))
        extra[:, 2] = extra[:, rng.integers(0, 2)]
        return v, np.concatenate([t, extra])
    if kind == "collinear":
        a, b = v[rng.integers(0, len(v), 12)], v[rng.integers(0, len(v), 12)]
        w = rng.uniform(-0.3, 1.3, (12, 1))
        w = a + w * (b - a) + rng.normal(size=(12, 3)) * 10.0 ** rng.uniform(-17, -5, (12, 1))
        k = len(v) + 3 * np.arange(12)[:, None] + np.arange(3)
        return np.concatenate([v, np.stack([a, b, w], 1).reshape(-1, 3)]), np.concatenate([t, k])
    return np.concatenate([v, [[3.0, 0, 0]]]), np.concatenate([t, [[len(v)] * 3]])  # a point


@pytest.mark.parametrize("kind", ["integers", "rounded", "repeated", "collinear", "point"])
@pytest.mark.parametrize("iso", [-0.5, 0.05, 0.6, 1.5])
def test_degenerate_meshes_equal_host(native, kind, iso):
    from visacd_gb300 import build
    build.build_host()
    import visacd_gb300.visacd as V
    for seed in range(8):
        rng = np.random.default_rng([seed, int(iso * 100) & 255])
        v, t = _mesh(kind, rng)
        t = np.ascontiguousarray(t, np.int32)
        scale = float(rng.uniform(4, 25)) / max(np.ptp(v, axis=0).max(), 1e-9)
        h = V._manifold_preprocess(v, t, scale, iso / scale)
        g = V._manifold_preprocess_gpu(v, t, scale, iso / scale)
        np.testing.assert_array_equal(g["triangles"], h["triangles"])
        np.testing.assert_array_equal(g["vertices"], h["vertices"])
