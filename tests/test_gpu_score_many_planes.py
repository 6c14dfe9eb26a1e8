"""Scoring of very many planes over few vertices, on both sides of the number of
plane groups that one launch of the kernels by vertex sides can hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 512])
@pytest.mark.parametrize("P", [65535 * 32, 65535 * 32 + 1])
def test_scores_past_the_grid_limit(ctx, orc, N, P):
    rng = np.random.default_rng(N + P)
    planes = rng.normal(size=(P, 4)).astype(np.float32)
    v = rng.normal(size=(N, 3)).astype(np.float32)
    e = rng.integers(0, N, (N + 3, 2)).astype(np.uint32)
    got, st = ctx.score_planes(planes, v, e)
    # the same planes in calls of a sixteenth, and some of them by the oracle
    want = np.concatenate([ctx.score_planes(part, v, e)[0] for part in np.array_split(planes, 16)])
    np.testing.assert_array_equal(got, want)
    assert st["argmax"] == int(np.argmax(want))
    some = np.concatenate([np.arange(100), np.arange(P - 100, P)])
    _, q, qexp, _ = orc.score_planes(planes[some], v, e)
    np.testing.assert_array_equal(got[some], np.ldexp(q.astype(np.float64), qexp))


def test_scores_without_room_for_the_sides(native, orc):
    """The table of sides of 2,000,000 planes and 512 vertices takes 320 MB; with less
    device memory left the call goes edge by edge."""
    torch = pytest.importorskip("torch")
    N, P = 512, 2000000
    rng = np.random.default_rng(3)
    planes = rng.normal(size=(P, 4)).astype(np.float32)
    v = rng.normal(size=(N, 3)).astype(np.float32)
    e = rng.integers(0, N, (N + 100, 2)).astype(np.uint32)
    ctx = native.Context(0)
    try:
        ctx.set_score_k(1)
        want, st = ctx.score_planes(planes, v, e)  # (also gets the room that way needs)
        ctx.set_score_k(0)
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        taken = torch.empty(free - (200 << 20), dtype=torch.uint8, device="cuda")
        try:
            got, sg = ctx.score_planes(planes, v, e)
        finally:
            del taken
            torch.cuda.empty_cache()
        np.testing.assert_array_equal(got, want)
        assert sg["argmax"] == st["argmax"]
        np.testing.assert_array_equal(ctx.score_planes(planes, v, e)[0], want)  # with room again
    finally:
        ctx.close()
