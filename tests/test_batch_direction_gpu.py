"""Batched BFS with bottom-up levels: depths and level counts equal one oracle
BFS per source.  Hub rows longer than a thread walks alone (29 in-edges) and
than a warp's step (128), graphs that begin inside a bitmap word, lanes whose
source sits in a small component or is unused, long tails after a dense part
(back to top-down), directed graphs, every lane-group width."""
import numpy as np
import pytest

import oracle
from graphreduce_gb300 import Batch
from graphreduce_gb300.graph import EdgeList

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(libgas):
    return libgas


def with_tail(el, n):
    """A path of n vertices hung on vertex 0, both directions."""
    a = np.concatenate([[0], np.arange(el.nV, el.nV + n - 1)]).astype(np.int32)
    b = np.arange(el.nV, el.nV + n, dtype=np.int32)
    return EdgeList(el.nV + n, np.concatenate([el.src, a, b]), np.concatenate([el.dst, b, a]))


def star(n):
    i = np.arange(1, n, dtype=np.int32)
    z = np.zeros(n - 1, np.int32)
    return EdgeList(n, np.concatenate([z, i]), np.concatenate([i, z]))


@pytest.fixture(scope="module")
def graphs():
    return [EdgeList.rmat(11, 16, seed=1), star(1001), EdgeList.rmat(9, 16, seed=2, symmetrize=False),
            with_tail(EdgeList.rmat(10, 24, seed=3), 300), EdgeList(5, *(np.zeros(0, np.int32),) * 2),
            EdgeList.erdos_renyi(3001, 24000, seed=4, symmetrize=True),
            EdgeList.rmat(8, 8, seed=5).with_grid_islands(7, 9)]


@pytest.mark.parametrize("lanes", [1, 2, 3, 7, 16, 19, 32])
@pytest.mark.parametrize("which", ["all", "one"])
def test_depths_and_levels(graphs, lanes, which):
    gs = graphs if which == "all" else graphs[:1]
    rng = np.random.default_rng(lanes)
    b = Batch()
    for el in gs:
        b.add_graph(el.nV, el.src, el.dst)
    b.build()
    for rep in range(2):  # the second run finds the first one's state
        srcs = np.stack([rng.integers(0, el.nV, lanes) for el in gs]).astype(np.int32)
        srcs[rng.random(srcs.shape) < 0.1] = -1
        if which == "all":
            srcs[3, 0] = gs[3].nV - 1  # from the tail's end
            srcs[6, -1] = gs[6].nV - 1  # an island
        r = b.run(bfs_sources=srcs)
        levels = 0
        for g, el in enumerate(gs):
            d = b.slice(r.depth, g)
            for l in range(lanes):
                if srcs[g, l] < 0:
                    assert np.all(d[:, l] == -1)
                    continue
                ref, it = oracle.bfs(el.nV, el.src, el.dst, int(srcs[g, l]))
                np.testing.assert_array_equal(d[:, l], ref, err_msg=f"graph {g} lane {l}")
                levels = max(levels, it)
        assert r.stats.bfs_iterations == max(0, levels - 1)
    b.close()
