"""The scoring autotuner's choices are the ones later calls use: planes per thread
where a call goes edge by edge, and whether it does."""
import numpy as np
import pytest

from visacd_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def _kernels(ctx, *call):
    best, used = 1e9, None
    for _ in range(4):
        ctx.set_timing(True)
        try:
            ctx.reset_times()
            ctx.score_planes(*call)
            k = ctx.kernel_times()
        finally:
            ctx.set_timing(False)
        names = [n for n in ("score_planes", "score_recheck_fp64", "plane_sides", "pack_edges") if k.get(n, (0, 0))[1]]
        best, used = min(best, sum(k[n][0] for n in names)), names
    return best, used


@pytest.mark.parametrize("N,E,P", [(2562, 30000, 592), (24576, 24576, 4096), (24000, 24100, 64), (4000, 3000, 700),
                                   (30000, 60000, 300)])
def test_later_calls_use_what_was_timed(native, N, E, P):
    ctx = native.Context(0)
    rng = np.random.default_rng(N)
    v = rng.normal(size=(N, 3)).astype(np.float32)
    e = rng.integers(0, N, (E, 2)).astype(np.uint32)
    planes = mg.random_planes(P, 3)
    want, _ = ctx.score_planes(planes, v, e)
    can = E >= N and N <= 24576
    before = ctx.launches
    best, ms = ctx.autotune_scoring(planes, v, e)
    # five launches a call either way, each choice twice
    assert ctx.launches - before == (50 if can else 40)
    assert best == (1, 2, 4, 8)[int(np.argmin(ms))]
    np.testing.assert_array_equal(ctx.score_planes(planes, v, e)[0], want)
    took, used = _kernels(ctx, planes, v, e)
    ctx.set_score_k(best)
    edges, by_edges = _kernels(ctx, planes, v, e)
    ctx.set_score_k(0)
    assert "plane_sides" not in by_edges
    if "plane_sides" in used:
        assert can and took <= 1.1 * edges + 2e-3
    else:
        assert took <= 1.1 * edges + 2e-3
    ctx.close()
