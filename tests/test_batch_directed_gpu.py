"""Batched BFS on directed CSRs whose last level holds only vertices without
out-edges: those get a level but form no frontier, so the largest level is one
above what a symmetric graph of the same number of frontiers would have. Levels
on both sides of every power of two, where that takes one more level plane."""
import numpy as np
import pytest

import oracle
from xbfs_b200 import Graph

pytestmark = pytest.mark.gpu

DEPTHS = [1, 2, 3, 4, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 254, 255, 256, 257]


def _csr(n, edges):
    e = np.array(sorted(edges), dtype=np.int64).reshape(-1, 2)
    beg = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(np.bincount(e[:, 0], minlength=n), out=beg[1:])
    return beg, e[:, 1].astype(np.int32)


def _chain(depth):
    """0 -> 1 -> ... -> depth: the last vertex is a sink."""
    return _csr(depth + 1, [(i, i + 1) for i in range(depth)])


def _broom(depth, leaves=67):
    """A chain whose last vertex but one links to `leaves` sinks."""
    return _csr(depth + leaves, [(i, i + 1) for i in range(depth - 1)] +
                [(depth - 1, depth + k) for k in range(leaves)])


def _check(beg, csr, srcs, words):
    r = Graph.from_csr(beg, csr).bfs_batch(srcs, words_per_vertex=words)
    mc = 0
    for i, s in enumerate(srcs):
        ref = oracle.bfs_queue(beg, csr, int(s))
        assert np.array_equal(r.levels[i], ref), f"source {s}: {np.nonzero(r.levels[i] != ref)[0][:8]}"
        mc += int(np.diff(beg)[ref >= 0].sum())
    assert r.edges_mc == mc // 2


@pytest.mark.parametrize("words", [1, 2, 4, 8])
@pytest.mark.parametrize("depth", DEPTHS)
def test_sinks_at_the_last_level(depth, words):
    beg, csr = _chain(depth)
    _check(beg, csr, np.array([0], dtype=np.int32), words)
    beg, csr = _broom(depth)
    _check(beg, csr, np.array([0], dtype=np.int32), words)
    # and among sources whose own last levels lie elsewhere, the sinks' included
    n = len(beg) - 1
    _check(beg, csr, (np.arange(64 * words - 3) * 7 % n).astype(np.int32), words)


@pytest.mark.parametrize("words", [1, 8])
def test_out_tree_of_sinks(words):
    depth, fan = 4, 5   # levels 0..4, the last one 625 sinks
    edges, level, n = [], [0], 1
    for _ in range(depth):
        nxt = []
        for u in level:
            for _ in range(fan):
                edges.append((u, n))
                nxt.append(n)
                n += 1
        level = nxt
    beg, csr = _csr(n, edges)
    _check(beg, csr, np.array([0, 1, n - 1], dtype=np.int32), words)
