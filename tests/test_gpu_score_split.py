"""How a scoring call is split (planes per thread, edge blocks per CTA) does not
show in its scores: at sizes on both sides of the blocks of 256 edges and of 256 K
planes the default split, every forced number of planes per thread and the
allocation-free entry give the same bits, and the sums of the cut edges' lengths
up to their quantisation (2^-23 of the largest length's power of two per edge)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [1, 255, 256, 257, 4661, 40000])
@pytest.mark.parametrize("P", [1, 255, 256, 257, 513, 1025, 2500])
def test_scores_do_not_depend_on_the_split(native, ctx, E, P):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(E * 10007 + P)
    v = rng.normal(size=(3000, 3)).astype(np.float32)
    e = rng.integers(0, len(v), (E, 2)).astype(np.uint32)
    n = rng.normal(size=(P, 3))
    planes = np.c_[n / np.linalg.norm(n, axis=1, keepdims=True), rng.uniform(-0.5, 0.5, P)].astype(np.float32)
    ctx.set_score_k(0)
    want = ctx.score_planes(planes, v, e)[0]
    try:
        for k in (1, 2, 4, 8):
            ctx.set_score_k(k)
            np.testing.assert_array_equal(ctx.score_planes(planes, v, e)[0], want)
    finally:
        ctx.set_score_k(0)
    d = [torch.from_numpy(a).cuda() for a in (planes, v, e.view(np.int32))]
    out, arg = torch.empty(P, dtype=torch.float64, device="cuda"), torch.empty(1, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream()
    p = [C.c_void_p(a.data_ptr()) for a in (*d, out, arg)]
    assert native.lib().visacd_score_planes_noalloc(p[0], P, p[1], len(v), p[2], C.c_int64(E), p[3], p[4],
                                                    C.c_void_p(st.cuda_stream)) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), want)
    # Lengths are FP32, decisions are of the FP64 values of the FP32 inputs.
    x = v.astype(np.float64)
    a, b = (planes[:, :3].astype(np.float64) @ x[e[:, i]].T + planes[:, 3:].astype(np.float64) for i in (0, 1))
    length = np.linalg.norm(x[e[:, 0]] - x[e[:, 1]], axis=1)
    eps = float(np.float32(1e-6))
    cut = ((a > eps) & (b < -eps)) | ((a < -eps) & (b > eps))
    unit = 2.0 ** (np.ceil(np.log2(max(length.max(), 1e-30))) - 22)
    assert np.abs(want - cut @ length).max() <= E * unit + 1e-6 * E
