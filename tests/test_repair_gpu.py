"""Isolated-node repair (dfs.h:63-137, 193-215) on given graphs, no build pass before it: against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(kind, r):
    """(rows, first unreached node): degree, then neighbours"""
    if kind == "few":      # one in 200 nodes has no in-edge: copies of the rows concerned
        n, R = 8000, 12
        g = np.zeros((n, R + 1), np.uint32)
        g[:, 0] = 6
        targets = np.setdiff1d(np.arange(n), np.arange(150, n, 200))
        g[:, 1:7] = r.choice(targets, (n, 6))
    elif kind == "most":   # the entry has no neighbours: every other node is unreached
        n, R = 5000, 8
        g = np.zeros((n, R + 1), np.uint32)
        g[:, 0] = r.integers(0, R + 1, n)
        g[:, 1:] = r.integers(0, n, (n, R))
        g[0, 0] = 0
    elif kind == "full":   # no row has room, but for a few far along: the last resort, a walk over all nodes
        n, R = 6000, 3
        g = np.zeros((n, R + 1), np.uint32)
        g[:, 0] = R
        g[:, 1:] = r.integers(0, n, (n, R))
        g[n - 40:, 0] = 1
    elif kind == "full_few":
        n, R = 20000, 6
        g = np.zeros((n, R + 1), np.uint32)
        g[:, 0] = R
        targets = np.setdiff1d(np.arange(n), np.arange(77, n, 997))
        g[:, 1:] = r.choice(targets, (n, R))
        g[n - 9:, 0] = 2
    else:                  # a chain of 700 levels with unreached nodes beside it
        n, R = 1100, 4
        g = np.zeros((n, R + 1), np.uint32)
        g[:700, 0], g[:700, 1] = 1, np.arange(1, 701)
        g[700:, 0], g[700:, 1:3] = 2, r.integers(0, n, (400, 2))
        g[699:701, 0] = 0
    g[:, 1:][np.arange(g.shape[1] - 1)[None, :] >= g[:, :1]] = 0
    return np.ascontiguousarray(g)


@pytest.mark.parametrize("kind", ["few", "most", "full", "full_few", "chain"])
def test_repair_matches_oracle(gpu_lib, oracle_lib, kind):
    from nbpg_gb300.index import Index
    r = np.random.default_rng(5)
    g0 = _graph(kind, r)
    n, R = g0.shape[0], g0.shape[1] - 1
    base = r.integers(0, 256, (n, 8)).astype(np.uint8)
    go, _, _, iso = oracle_lib.build_graph("u8", "l2", base, R=R, L=16, VL=24, num_split=0, num_passes=0, graph=g0)
    idx = Index(base, "u8", "l2", max_degree=R, graph=g0)
    st, _, _ = idx.build_vamana(L=16, VL=24, num_split=0, num_passes=0)
    g = idx.get_graph()
    assert st.isolated == iso > 0
    live = np.arange(R)[None, :] < go[:, :1]
    assert np.array_equal(g[:, 0], go[:, 0]) and np.array_equal(g[:, 1:][live], go[:, 1:][live])
