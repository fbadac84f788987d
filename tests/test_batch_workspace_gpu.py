"""Batched calls share pooled workspaces: a graph that needs more of a buffer
than the one before it must find it cleared, wherever the larger one lies."""
import ctypes
import gc

import numpy as np
import pytest

import oracle
from xbfs_b200 import Graph

pytestmark = pytest.mark.gpu


def _symmetric(n, pairs):
    e = np.array(pairs, dtype=np.int64)
    e = np.concatenate([e, e[:, ::-1]])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    beg = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(np.bincount(e[:, 0], minlength=n), out=beg[1:])
    return beg, e[:, 1].astype(np.int32)


class _OnesInFreedMemory:
    """Small device allocations, filled with ones and freed, but for a few that
    keep their pages mapped: what the next small allocations of the process get."""

    def __enter__(self):
        cuda = self.cuda = ctypes.CDLL("libcuda.so.1")
        ptrs = []
        for _ in range(2000):
            p = ctypes.c_uint64(0)
            assert cuda.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(512)) == 0
            ptrs.append(p)
            assert cuda.cuMemsetD8_v2(p, ctypes.c_ubyte(0xFF), ctypes.c_size_t(512)) == 0
        assert cuda.cuCtxSynchronize() == 0
        self.kept = ptrs[::250]
        for p in ptrs:
            if p not in self.kept:
                assert cuda.cuMemFree_v2(p) == 0

    def __exit__(self, *exc):
        for p in self.kept:
            assert self.cuda.cuMemFree_v2(p) == 0


@pytest.mark.parametrize("words", [1, 8])
def test_hubs_after_a_graph_without_hubs(words):
    gc.collect()  # handles of other tests: with the last one go the idle workspaces
    hubs, leaves = 6 if words == 8 else 50, 1100
    n = hubs + leaves
    plain = _symmetric(n, [(i, i + 1) for i in range(n - 1)])
    # every leaf on every hub: lists of 1100 edges, two chunks each
    hubby = _symmetric(n, [(h, hubs + k) for h in range(hubs) for k in range(leaves)])
    Graph.from_csr(*plain).bfs(0)
    with _OnesInFreedMemory():
        g0, g1 = Graph.from_csr(*plain), Graph.from_csr(*hubby)
        srcs = (np.arange(5) * 201).astype(np.int32)
        for g, (beg, csr) in ((g0, plain), (g1, hubby), (g0, plain), (g1, hubby)):
            r = g.bfs_batch(srcs, words_per_vertex=words, direction="bu")
            for i, s in enumerate(srcs):
                ref = oracle.bfs_queue(beg, csr, int(s))
                assert np.array_equal(r.levels[i], ref), f"source {s}: {np.nonzero(r.levels[i] != ref)[0][:8]}"
