"""BVHs used by another context than the one they were built on: a build from
host arrays is left running on its own context's stream, so whatever reads it
from another stream has to wait for it first."""
import numpy as np
import pytest

from visacd_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def test_batch_with_a_grid_over_another_contexts_cage(native, ctx):
    """A part of more than 2^22 pairs, whose cage gets a free-space grid inside the
    call: the cage is the last of several builds queued on its context when the
    other context takes it. The edges are those of the traversal alone, in the
    first call and (with the grid the BVH keeps) in a later one."""
    v, _ = mg.displaced_blob(5, seed=6)
    pts = np.ascontiguousarray(v[:3200], np.float32)
    none = np.zeros((0, 3), np.int32)
    cage = mg.offset_cage(*mg.displaced_blob(6, seed=6), 0.03)
    other = native.Context(0)
    sb = ctx.bvh(pts, none)
    builds = [other.bvh(*cage) for _ in range(8)]
    cb = builds[-1]
    first = ctx.visibility_batch([(pts, sb, cb, None)])[0][0]
    assert ctx.visibility(pts, sb, cb)[1]["pairs_tested"] == 3200 * 3199 // 2 >= 1 << 22
    assert ctx.vis_trace_counts()[0] > 0  # the walk is in use
    later = ctx.visibility_batch([(pts, sb, cb, None)])[0][0]
    ctx.set_vis_trace(False)
    try:
        want = ctx.visibility_batch([(pts, sb, cb, None)])[0][0]
    finally:
        ctx.set_vis_trace(True)
    assert len(want) > 0
    np.testing.assert_array_equal(first, want)
    np.testing.assert_array_equal(later, want)
    for b in builds:
        b.close()
    sb.close()
    other.close()


@pytest.mark.parametrize("level", [0, 2, 6])
def test_info_of_a_bvh_whose_context_went(native, ctx, level):
    mesh = mg.displaced_blob(level, seed=3)
    other = native.Context(0)
    kept, asked = other.bvh(*mesh), other.bvh(*mesh)
    want = asked.info()
    other.close()
    assert kept.info() == want and asked.info() == want
    again = ctx.bvh(*mesh)
    assert again.info() == want
    for b in (kept, asked, again):
        b.close()


def test_info_takes_little_time(ctx):
    """The depth of 81,920 triangles right after the build, the median of eleven:
    0.1 ms; 0.86 with the records brought to the host and walked there."""
    import time
    mesh = mg.displaced_blob(6, seed=3)
    took = []
    for _ in range(11):
        b = ctx.bvh(*mesh)
        ctx.synchronize()
        t0 = time.perf_counter()
        depth = b.info()[1]
        took.append(time.perf_counter() - t0)
        assert 17 <= depth <= 47
        b.close()
    assert np.median(took) < 4e-4


@pytest.mark.parametrize("call", ["visibility", "batch", "graph"])
def test_a_blocking_context_sleeps_through_anothers_build(native, call):
    """A context that waits blocking (many contexts sharing the cores) also waits so
    for a build on another context's stream, here behind 0.3 s of other work: the
    thread's own time is a small part of the wait."""
    import time
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    other, waiting = native.Context(0, stream=stream.cuda_stream), native.Context(0)
    assert native.lib().visacd_ctx_set_blocking_wait(waiting.handle, 1) == 0
    pts = mg.displaced_blob(1, seed=2)[0]
    cage, none = mg.displaced_blob(2, seed=3), np.zeros((0, 3), np.int32)
    planes = np.array([[1.0, 0, 0, 0]], np.float32)
    run = {"visibility": lambda a, b: waiting.visibility(pts, a, b)[0],
           "batch": lambda a, b: waiting.visibility_batch([(pts, a, b, None)])[0][0],
           "graph": lambda a, b: native.Batch(waiting, [(pts, a, b, planes)]).close()}[call]
    a, b = other.bvh(pts, none), other.bvh(*cage)
    want = run(a, b)  # first-call costs
    with torch.cuda.stream(stream):
        torch.cuda._sleep(600_000_000)  # a kernel of some 0.3 s
    c = other.bvh(*cage)
    t0, c0 = time.perf_counter(), time.thread_time()
    got = run(a, c)
    wall, cpu = time.perf_counter() - t0, time.thread_time() - c0
    np.testing.assert_array_equal(got, want)
    assert wall > 0.1  # it did wait
    assert cpu < 0.3 * wall
    for x in (a, b, c):
        x.close()
    waiting.close()
    other.close()


@pytest.mark.parametrize("which", ["part", "cage"])
def test_a_batch_refuses_a_bvh_whose_context_went(native, ctx, which):
    v, t = mg.displaced_blob(1, seed=2)
    cage = mg.offset_cage(v, t, 0.05)
    other = native.Context(0)
    a = (other if which == "part" else ctx).bvh(v, t)
    b = (other if which == "cage" else ctx).bvh(*cage)
    other.close()
    with pytest.raises(native.VisacdError):
        native.Batch(ctx, [(v, a, b, np.array([[1.0, 0, 0, 0]], np.float32))]).close()
    a.close()
    b.close()
