"""Per-level records of runs of small levels that end at any level of the ring in
which the records are handed over, with each policy's pace."""
import numpy as np
import pytest

from xbfs_b200 import Graph, learned

pytestmark = pytest.mark.gpu


def _cycle(n):
    """Two vertices a level, one at the end (n even)."""
    i = np.arange(n)
    nbr = np.sort(np.stack([(i - 1) % n, (i + 1) % n], 1), axis=1)
    return np.arange(n + 1, dtype=np.int64) * 2, nbr.ravel().astype(np.int32)


@pytest.mark.parametrize("policy", ["heuristic", "mlp"])
def test_records_of_runs_of_every_length(policy):
    if policy == "mlp":
        learned.install(learned.load()[0])
    try:
        for last in list(range(60, 92)) + [96, 112, 128, 144, 160]:
            g = Graph.from_csr(*_cycle(2 * last))
            for _ in range(10):
                r = g.bfs(0, policy=policy, trace=True)
                assert [t["n_f"] for t in r.trace] == [1] + [2] * (last - 1) + [1]
                assert [t["m_f"] for t in r.trace] == [2] + [4] * (last - 1) + [2]
    finally:
        if policy == "mlp":
            learned.install(None)
