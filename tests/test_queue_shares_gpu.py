"""Small queues shared by grids of a few CTAs: queues on both sides of 32 entries a
CTA, where some shares are one entry larger than others."""
import numpy as np
import pytest

import oracle
from xbfs_b200 import Graph

pytestmark = pytest.mark.gpu


def _broom(n):
    """A vertex with n neighbours, of which the last third have two leaves each: level
    1 is a queue of n vertices whose edges gather at one end."""
    heavy = np.arange(n - n // 3, n) + 1
    e = np.stack([np.zeros(n, dtype=np.int64), np.arange(n) + 1], 1)
    e = np.concatenate([e, np.stack([np.repeat(heavy, 2), n + 1 + np.arange(2 * len(heavy))], 1)])
    e = np.concatenate([e, e[:, ::-1]])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    V = n + 1 + 2 * len(heavy)
    beg = np.zeros(V + 1, dtype=np.int64)
    np.cumsum(np.bincount(e[:, 0], minlength=V), out=beg[1:])
    return beg, e[:, 1].astype(np.int32)


@pytest.mark.parametrize("blocks", [1, 2, 3, 7, 16, 25, 31, 32, 40])
@pytest.mark.parametrize("policy", ["heuristic", "beamer", "forced"])
def test_shares_of_32_entries_and_one_more(blocks, policy):
    kw = {"policy": policy}
    if policy == "forced":
        kw["forced"] = ["td_queue"]
    for n in sorted({32 * blocks - 1, 32 * blocks, 32 * blocks + 1, 32 * blocks + blocks // 2 + 1, 33 * blocks - 1,
                        33 * blocks, 33 * blocks + 1}):
        beg, csr = _broom(n)
        ref = oracle.bfs_queue(beg, csr, 0)
        g = Graph.from_csr(beg, csr)
        for grid_dim in (blocks, 0):
            r = g.bfs(0, want_parents=True, grid_dim=grid_dim, **kw)
            assert np.array_equal(r.levels, ref), (n, grid_dim, np.nonzero(r.levels != ref)[0][:8])
            assert r.reached == len(ref) and oracle.check_tree(beg, csr, 0, r.levels, r.parents) == 0
