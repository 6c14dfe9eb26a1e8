"""Sampled Hausdorff terms where samples lie at exactly equal distances at the
tenth place: the ones that count are the first in the order of the search (rings
of cells around the query, in a ring by cell), and such a query takes about as long
as another."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _visit_order(x, q):
    """Ring and cell of each sample in the grid the samples get (about two samples
    per occupied cell, at most 160 cells per axis)."""
    lo, hi = x.min(0), x.max(0)
    d = hi - lo
    h = max(np.sqrt(max(d[0] * d[1] + d[1] * d[2] + d[2] * d[0], 1e-30) * 2.0 / len(x)), d.max() / 160.0)
    dim = np.maximum(1, np.ceil(d / h).astype(int) + 1)
    cell = lambda p: np.clip(np.floor((p - lo) / h).astype(int), 0, dim - 1)
    c, cq = cell(x), cell(q)
    return list(zip(np.abs(c - cq).max(1), c[:, 2], c[:, 1], c[:, 0]))


@pytest.mark.parametrize("seed", range(12))
def test_equal_distances_count_in_the_order_of_the_search(ctx, seed):
    rng = np.random.default_rng(seed)
    q = rng.integers(-8, 9, 3) * 0.125
    corner = np.array(list(itertools.product([-1.0, 1.0], repeat=3)))
    axes = np.concatenate([np.eye(3), -np.eye(3)])
    x = np.concatenate([0.5 * axes[[0, 1, 3, 4]], corner, 2.5 * axes]) + q  # ranks 0-3, 4-11 (equal), 12-17
    dist = np.concatenate([np.full(4, 9.0), 5.0 + 0.25 * rng.permutation(8), np.full(6, 9.5)])
    order = rng.permutation(len(x))
    x, dist = x[order], dist[order]
    # each sample's own triangle, parallel to z over the query at its distance
    v = np.concatenate([q + [[-30.0, -30.0, z], [30.0, -30.0, z], [0.0, 30.0, z]] for z in dist])
    t = np.arange(3 * len(x), dtype=np.int32).reshape(-1, 3)
    small = q + np.array([[0.1, 0, 0], [0, 0.1, 0], [-0.1, -0.1, 0]])
    rank = sorted(range(len(x)), key=lambda i: (round(float(((x[i] - q) ** 2).sum()), 9), _visit_order(x, q)[i]))
    want = dist[rank[:10]].min()
    got = ctx.face_hausdorff(small, np.array([[0, 1, 2]], np.int32), q[None], np.zeros(1, np.int32),
                             v, t, x, np.arange(len(x), dtype=np.int32))
    assert abs(got - want) <= 1e-11


def _lattice(n, z, jitter, seed):
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(np.arange(n), np.arange(n), indexing="ij"), -1).reshape(-1, 2)
    v = np.c_[g / n, np.full(n * n, z)] + rng.uniform(-jitter, jitter, (n * n, 3))
    i = (np.arange(n - 1)[:, None] * n + np.arange(n - 1)).ravel()
    t = np.r_[np.c_[i, i + 1, i + n], np.c_[i + 1, i + n + 1, i + n]].astype(np.int32)
    ids = np.zeros(n * n, np.int32)
    ids[t.ravel()] = np.repeat(np.arange(len(t)), 3)
    return v, t, v.copy(), ids


def test_ties_take_no_longer(ctx):
    """Two lattices of samples: every query has ties at the tenth place. Kernel
    times, the least of eight calls: 2.1 times those of jittered lattices (of which
    fewer queries need evaluation), 11 times when a tie costs a warp's time."""
    def kernels(jitter):
        a, b = _lattice(128, 0.0, jitter, 1), _lattice(128, 0.005, jitter, 2)
        best = 1e9
        for _ in range(8):
            ctx.set_timing(True)
            try:
                ctx.reset_times()
                assert abs(ctx.face_hausdorff(*a, *b) - 0.005) <= 4 * jitter + 1e-9
                k = ctx.kernel_times()
            finally:
                ctx.set_timing(False)
            best = min(best, k["hd_head"][0] + k["hd_query"][0])
        return best

    assert kernels(0.0) <= 4 * kernels(1e-6)
