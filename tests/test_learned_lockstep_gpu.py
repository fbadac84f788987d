"""The learned switch in runs of small levels that several CTAs share: each CTA
decides for itself, so all must decide alike at every level. Networks whose
choice flips within such runs (random weights, the bias set so that a share of
the levels leaves the queue-based top-down), weights beyond what the certificate
of a reused decision can carry, and the shipped ones: right levels, no wait that
runs out, and the network's own choice at every level that is no tie."""
import numpy as np
import pytest

from xbfs_b200 import Graph, learned

pytestmark = pytest.mark.gpu


def _grid_levels(w, h, src):
    i = np.arange(w * h)
    return (np.abs(i % w - src % w) + np.abs(i // w - src // w)).astype(np.int32)


def _features(trace):
    ids = {"td_queue": 0, "td_scan": 1, "bu": 2}
    rows = [dict(t, strategy_id=ids[t["strategy"]]) for t in trace]
    return learned.features_from_trace(rows), [r["strategy_id"] for r in rows]


@pytest.mark.parametrize("size", [(900, 700), (64, 3000)])
@pytest.mark.parametrize("share", [0.0, 0.02, 0.3])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_networks_that_leave_runs(size, share, seed):
    w, h = size
    src = w * (h // 2) + w // 3
    ref = _grid_levels(w, h, src)
    g = Graph.grid(w, h)
    feats, _ = _features(g.bfs(src, trace=True).trace)
    net = learned.init_weights(feats, seed)
    lg = learned.logits(net, feats)
    net[-3] += np.float32(np.quantile(np.max(lg[:, 1:], axis=1) - lg[:, 0], 1.0 - share))
    learned.install(net)
    try:
        for _ in range(3):
            r = g.bfs(src, policy="mlp", trace=True)
            assert np.array_equal(r.levels, ref)
            feats, took = _features(r.trace)
            lg = learned.logits(net, feats)
            top = np.sort(lg, axis=1)
            clear = top[:, 2] - top[:, 1] > 1e-3   # elsewhere a tie within float noise
            assert np.array_equal(np.array(took)[clear], np.argmax(lg, axis=1)[clear])
    finally:
        learned.install(None)


@pytest.mark.parametrize("scale", [1e10, 1e13, float("inf"), float("nan")])
def test_weights_beyond_the_certificate(scale):
    w, h, src = 900, 700, 315300
    g = Graph.grid(w, h)
    feats, _ = _features(g.bfs(src, trace=True).trace)
    net = learned.init_weights(feats, 3)
    with np.errstate(invalid="ignore"):
        net[16:] *= np.float32(scale)
    learned.install(net)
    try:
        assert np.array_equal(g.bfs(src, policy="mlp").levels, _grid_levels(w, h, src))
    finally:
        learned.install(None)
