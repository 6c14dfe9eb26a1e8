"""Visibility calls with points and mask in device memory: the edges and counts of
the same call from host arrays, and the same work for them (a few new points among
many are few pairs, which need no free-space walk and no reach table)."""
import ctypes as C

import numpy as np
import pytest

from visacd_gb300 import meshgen as mg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _device(native, ctx, pts, mask, sb, cb):
    p, m = torch.from_numpy(pts).cuda(), torch.from_numpy(mask).cuda()
    torch.cuda.synchronize()
    ne, st = C.c_int64(), native.VisStats()
    assert native.lib().visacd_visibility(ctx.handle, C.c_void_p(p.data_ptr()), len(pts), C.c_void_p(m.data_ptr()), 1,
                                          sb.handle, cb.handle, C.byref(ne), C.byref(st)) == 0
    out = np.empty((ne.value, 2), np.uint32)
    assert native.lib().visacd_visibility_edges(ctx.handle, native._ptr(out), ne.value) == 0
    return out, st.as_dict()


@pytest.mark.parametrize("n,new", [(2, 1), (33, 0), (33, 33), (700, 5), (3000, 100), (3300, 1700), (20000, 30),
                                   (140000, 2)])
def test_device_mask_equals_host_mask(native, ctx, n, new):
    rng = np.random.default_rng(n + new)
    pts = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    mask = np.zeros(n, np.uint8)
    mask[rng.permutation(n)[:new]] = rng.integers(1, 256, new)
    sb, cb = ctx.bvh(pts, np.zeros((0, 3), np.int32)), ctx.bvh(*mg.displaced_blob(3, seed=2))
    want, ws = ctx.visibility(pts, sb, cb, is_new=mask)
    walked = ctx.vis_trace_counts()
    got, gs = _device(native, ctx, pts, mask, sb, cb)
    np.testing.assert_array_equal(got, want)
    assert gs == ws
    assert ws["pairs_tested"] == n * (n - 1) // 2 - (n - new) * (n - new - 1) // 2
    assert ctx.vis_trace_counts() == walked
    assert walked[0] == 0 or ws["pairs_tested"] >= 1 << 22
    sb.close()
    cb.close()
