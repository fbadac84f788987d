"""Runs of small top-down levels (a few CTAs keep the frontier in shared memory
while the others wait): levels, parents, per-level statistics and totals on deep
graphs whose frontiers start, leave and re-enter such runs in every way: one CTA
or several, too many edges, vertices of too large a degree, more edges than fit,
shares that become uneven, dead ends of a directed CSR."""
import numpy as np
import pytest

import oracle
from xbfs_b200 import Graph, gen_grid_host, learned

pytestmark = pytest.mark.gpu


def _csr(pairs, V, directed=False):
    e = np.array(pairs, dtype=np.int64).reshape(-1, 2)
    if not directed:
        e = np.concatenate([e, e[:, ::-1]])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    beg = np.zeros(V + 1, dtype=np.int64)
    np.cumsum(np.bincount(e[:, 0], minlength=V), out=beg[1:])
    return beg, e[:, 1].astype(np.int32)


def _path(n):
    return _csr([(i, i + 1) for i in range(n - 1)], n)


def _hubs_on_a_path():
    """Leaves on a path: vertices of more edges than the small bin holds."""
    pairs, V = [(i, i + 1) for i in range(599)], 600
    for at, deg in ((40, 31), (60, 33), (120, 300), (200, 5000), (201, 40), (420, 64)):
        pairs += [(at, V + k) for k in range(deg)]
        V += deg
    return _csr(pairs, V)


def _path_into_trees(fan):
    """A path, then a tree of the given fan-out: a frontier that outgrows a run
    in one level, then a long path on from one leaf."""
    pairs, V, level = [(i, i + 1) for i in range(29)], 30, [29]
    while len(level) < 20000:
        nxt = []
        for u in level:
            nxt += range(V, V + fan)
            pairs += [(u, v) for v in range(V, V + fan)]
            V += fan
        level = nxt
    pairs += [(level[0], V)] + [(i, i + 1) for i in range(V, V + 199)]
    return _csr(pairs, V + 200)


def _directed_grid(w, h):
    """Edges right and down only; every seventh vertex leads nowhere."""
    idx = np.arange(w * h)
    pairs = [np.stack([idx[(idx % w) < w - 1], idx[(idx % w) < w - 1] + 1], 1), np.stack([idx[:-w], idx[:-w] + w], 1)]
    e = np.concatenate(pairs)
    return _csr(e[(e[:, 0] % 7 != 3) | (e[:, 0] < w)], w * h, directed=True)


def _fan_of_paths(n, length):
    """One vertex with n paths, joined crosswise near the end."""
    pairs = []
    for k in range(n):
        c = [0] + list(range(1 + k * length, 1 + (k + 1) * length))
        pairs += list(zip(c[:-1], c[1:]))
    pairs += [(1 + k * length + length - 1, 1 + ((k * 7 + 1) % n) * length + length // 2) for k in range(n)]
    return _csr(pairs, 1 + n * length)


GRAPHS = {
    "path": (lambda: _path(3001), 1500),
    "grid_one_cta": (lambda: gen_grid_host(90, 70), 333),
    "grid": (lambda: gen_grid_host(701, 601), 70000),
    "grid_from_corner": (lambda: gen_grid_host(1500, 300), 0),
    "hubs": (_hubs_on_a_path, 0),
    "tree8": (lambda: _path_into_trees(8), 0),
    "tree31": (lambda: _path_into_trees(31), 0),
    "directed": (lambda: _directed_grid(301, 257), 0),
    "fan": (lambda: _fan_of_paths(700, 60), 0),
}


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("policy", ["heuristic", "beamer", "mlp", "forced", "mixed"])
def test_runs_of_small_levels(name, policy):
    make, src = GRAPHS[name]
    beg, csr = make()
    ref = oracle.bfs_queue(beg, csr, src)
    deg = np.diff(beg)
    depth = int(ref.max()) + 1
    kw = {"policy": policy}
    if policy == "forced":
        kw["forced"] = ["td_queue"]
    if policy == "mixed":  # every 37th level something else
        kw = {"policy": "forced", "forced": [("td_scan", "bu")[(i // 37) % 2] if i % 37 == 36 else "td_queue"
                                             for i in range(depth)]}
    if policy == "mlp":
        learned.install(learned.load()[0])
    try:
        g = Graph.from_csr(beg, csr)
        for grid_dim in (0, 1, 5, 40):
            r = g.bfs(src, want_parents=grid_dim != 5, trace=True, grid_dim=grid_dim, **kw)
            assert np.array_equal(r.levels, ref), np.nonzero(r.levels != ref)[0][:8]
            if r.parents is not None:
                assert oracle.check_tree(beg, csr, src, r.levels, r.parents) == 0
            assert r.depth == depth and r.reached == int((ref >= 0).sum())
            assert r.edges_mc == int(deg[ref >= 0].sum()) // 2 and sum(r.strategies.values()) == depth
            assert len(r.trace) == depth
            n_f = np.bincount(ref[ref >= 0], minlength=depth)
            m_f = np.bincount(ref[ref >= 0], weights=deg[ref >= 0], minlength=depth).astype(np.int64)
            assert [t["n_f"] for t in r.trace] == n_f.tolist()
            assert [t["m_f"] for t in r.trace] == m_f.tolist()
    finally:
        if policy == "mlp":
            learned.install(None)


def test_runs_over_many_sources():
    beg, csr = gen_grid_host(400, 300)
    g = Graph.from_csr(beg, csr)
    srcs = np.arange(0, g.V, 9973, dtype=np.int32)
    r = g.bfs_many(srcs)
    for s, lv in zip(srcs, r.levels):
        assert np.array_equal(lv, oracle.bfs_queue(beg, csr, int(s)))
