"""Batched multi-source BFS (64 sources per uint64 word): every per-source
level array bit-exact against the serial CPU BFS, for every word width,
direction choice, duplicate sources, deep graphs (two-byte level rows) and
host or device output."""
import numpy as np
import pytest

import oracle
from tests.conftest import hand_graphs
from xbfs_b200 import Graph, gen_er_host, gen_grid_host, gen_rmat_host, pick_sources

pytestmark = pytest.mark.gpu


def check_batch(g, beg, csr, srcs, **kw):
    r = g.bfs_batch(srcs, **kw)
    mc = 0
    for i, s in enumerate(srcs):
        ref = oracle.bfs_queue(beg, csr, int(s))
        assert np.array_equal(r.levels[i], ref), f"source #{i} ({s}) differs at {np.nonzero(r.levels[i] != ref)[0][:8]}"
        mc += int(np.diff(beg)[ref >= 0].sum())
    assert r.edges_mc == mc // 2  # Graph500 m_c summed over sources
    return r


@pytest.mark.parametrize("words", [1, 2, 4, 8])
@pytest.mark.parametrize("direction", [None, "td", "bu"])
def test_rmat_all_widths_and_directions(words, direction):
    beg, csr = gen_rmat_host(12, 16, 3)
    g = Graph.from_csr(beg, csr)
    srcs = pick_sources(beg, 64 * words - 7, 3)  # a partial last word
    check_batch(g, beg, csr, srcs, words_per_vertex=words, direction=direction)


def test_512_sources_multiple_passes_and_duplicates():
    beg, csr = gen_rmat_host(13, 8, 5)
    g = Graph.from_csr(beg, csr)
    srcs = np.concatenate([pick_sources(beg, 300, 5), pick_sources(beg, 300, 5)[:40]])  # duplicates
    check_batch(g, beg, csr, srcs, words_per_vertex=2)   # 5 passes of 128
    check_batch(g, beg, csr, srcs[:512])                 # auto width


def test_hand_graphs_including_isolated_sources():
    for name, (beg, csr) in hand_graphs().items():
        g = Graph.from_csr(beg, csr)
        n = len(beg) - 1
        srcs = np.arange(n, dtype=np.int32) if n <= 64 else np.arange(0, n, max(1, n // 60), dtype=np.int32)
        check_batch(g, beg, csr, srcs, words_per_vertex=1)


def test_deep_grid_uses_wide_level_rows():
    beg, csr = gen_grid_host(300, 3)   # diameter ~ 301 > 254
    g = Graph.from_csr(beg, csr)
    check_batch(g, beg, csr, np.array([0, 450, 899, 1], dtype=np.int32), words_per_vertex=1)


def test_er_and_device_output():
    import torch
    beg, csr = gen_er_host(30000, 8.0, 2)
    g = Graph.from_csr(beg, csr)
    srcs = pick_sources(beg, 200, 2)
    out = torch.empty((len(srcs), g.V), dtype=torch.int32, device="cuda:0")
    g.bfs_batch(srcs, levels=out)
    torch.cuda.synchronize()
    lv = out.cpu().numpy()
    for i in (0, 57, 199):
        assert np.array_equal(lv[i], oracle.bfs_queue(beg, csr, int(srcs[i])))


def _stars_and_path(degrees, path):
    """Hubs of the given degrees whose leaves are shared (leaf k hangs on every
    hub of degree > k), a path hanging on the first leaf, a separate pair and an
    isolated last vertex: list lengths on both sides of each way a bottom-up
    search is split, sources whose component is soon exhausted, a deep tail."""
    nh, nl = len(degrees), max(degrees)
    pairs = [(h, nh + k) for h, d in enumerate(degrees) for k in range(d)]
    first = nh + nl
    chain = [nh] + list(range(first, first + path))
    pairs += list(zip(chain[:-1], chain[1:]))
    a = first + path
    pairs.append((a, a + 1))
    V = a + 3
    e = np.array(pairs, dtype=np.int64)
    e = np.concatenate([e, e[:, ::-1]])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    beg = np.zeros(V + 1, dtype=np.int64)
    np.cumsum(np.bincount(e[:, 0], minlength=V), out=beg[1:])
    return beg, e[:, 1].astype(np.int32)


@pytest.mark.parametrize("words", [1, 2, 4, 8])
@pytest.mark.parametrize("direction", [None, "td", "bu"])
def test_split_lists_and_level_planes(words, direction):
    beg, csr = _stars_and_path([64, 65, 1024, 1025, 2048, 5000], 300)   # 300 levels: planes past the low eight
    g = Graph.from_csr(beg, csr)
    n = 64 * words
    srcs = np.random.default_rng(words).integers(0, g.V, size=n - 3).astype(np.int32)
    srcs = np.concatenate([srcs, [0, g.V - 1, g.V - 3]]).astype(np.int32)
    check_batch(g, beg, csr, srcs, words_per_vertex=words, direction=direction)


@pytest.mark.parametrize("depth", [1, 2, 3, 4, 7, 8, 9, 127, 128, 129, 255, 256, 257])
def test_levels_at_plane_borders(depth):
    n = depth + 1
    beg = np.concatenate([[0], np.cumsum([1] + [2] * (n - 2) + [1])]).astype(np.int64)
    csr = np.concatenate([[1]] + [[i - 1, i + 1] for i in range(1, n - 1)] + [[n - 2]]).astype(np.int32)
    g = Graph.from_csr(beg, csr)
    for direction in ("td", "bu"):
        check_batch(g, beg, csr, np.array([0, n // 2], dtype=np.int32), direction=direction)


def test_graphs_of_other_sizes_in_turn():
    made = [gen_rmat_host(11, 8, 1), gen_rmat_host(14, 24, 2), gen_er_host(3001, 8.0, 3), gen_grid_host(17, 19)]
    graphs = [Graph.from_csr(*m) for m in made]
    for rep, n in enumerate((512, 3, 130)):
        for g, (beg, csr) in zip(graphs, made):
            check_batch(g, beg, csr, pick_sources(beg, n, rep))


def test_directed_rows():
    rng = np.random.default_rng(4)
    deg = rng.integers(0, 9, size=3001)
    beg = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    csr = rng.integers(0, 3001, size=int(beg[-1])).astype(np.int32)
    g = Graph.from_csr(beg, csr)
    for words in (1, 8):
        r = g.bfs_batch(np.arange(200, dtype=np.int32), words_per_vertex=words)
        for i in range(200):
            assert np.array_equal(r.levels[i], oracle.bfs_queue(beg, csr, i))
