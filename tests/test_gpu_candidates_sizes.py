"""Candidate planes at the edges of the tiles of the similarity test (256
candidates) and of the states kept in shared memory (32,768): a prefix of the
draws keeps a prefix of the oracle's planes, bit for bit."""
import numpy as np
import pytest

from visacd_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def _edges(level, seed):
    v, t = mg.displaced_blob(level, seed=seed)
    e = np.sort(np.concatenate([t[:, [0, 1]], t[:, [1, 2]], t[:, [2, 0]]]), axis=1)
    return v, np.unique(e, axis=0).astype(np.uint32)


def _prefix(draws, unique):
    first = np.sort(np.unique(draws, return_index=True)[1])
    return draws[:first[unique - 1] + 1]


@pytest.mark.parametrize("level,num,sizes", [
    (4, 600, (1, 2, 255, 256, 257, 511, 512, 513, 1025, 1537, 2305)),
    (6, 8000, (32767, 32768, 32769, 33100)),
])
def test_candidate_counts_at_edges(ctx, orc, level, num, sizes):
    v, e = _edges(level, 3)
    want, draws, used = orc.candidate_planes_with_draws(v, e, num, 11)
    got, got_used = ctx.candidate_planes(v, e, draws, num)
    np.testing.assert_array_equal(got, want)
    assert got_used == used
    assert len(np.unique(draws)) >= max(sizes)
    kept = 0
    for n in sizes:
        d = _prefix(draws, n)
        got, got_used = ctx.candidate_planes(v, e, d, num)
        assert kept <= len(got) <= n and (len(got) == num or got_used == len(d))
        np.testing.assert_array_equal(got, want[:len(got)])
        kept = len(got)
