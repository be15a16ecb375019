"""The precision PageRank gather at its edges: rows around the tile's 256
in-edges and the lane's 8, rows without in-edges, edge counts around whole
tiles, and graphs large enough for the hot sources' copy, against FP64."""
from contextlib import closing

import numpy as np
import pytest
from scipy.sparse import csr_matrix

from graphreduce_gb300 import GASEngineGPU
from graphreduce_gb300.engine import initial_vertex_data
from graphreduce_gb300.graph import EdgeList

pytestmark = pytest.mark.gpu

D, TOL = 0.85, 1e-7
# the FP32 iteration: contribution, sum, product and rank are rounded, at most
# 8 + 2 additions deep between two-sums, 16 roundings of 2^-24 of ranks that
# sum to at most 1, carried on by the factor 1 / (1 - D); and either side may
# stop one step of at most TOL, carried on alike, before the other
BOUND = (16 * 2.0 ** -24 + TOL) / (1 - D)


@pytest.fixture(scope="module", autouse=True)
def _built(libgas):
    return libgas


def reference(el, start, base, steps=100000):
    outdeg = np.bincount(el.src, minlength=el.nV)
    inv = np.divide(1.0, outdeg, where=outdeg > 0, out=np.zeros(el.nV))
    m = csr_matrix((inv[el.src], (el.dst, el.src)), shape=(el.nV, el.nV))
    r = start
    for _ in range(steps):
        new = base + D * (m @ r)
        done = np.abs(new - r).sum() <= TOL
        r = new
        if done:
            return r
    raise AssertionError("no convergence")


def check(el, hot=None, seeds=()):
    with closing(GASEngineGPU("pagerank")) as eng:
        vd = initial_vertex_data("pagerank", el.nV, 0, el.out_degree())
        eng.setGraph(el.nV, vd, el.nE, None, el.src, el.dst)
        one = np.ones(el.nV)
        cases = [(lambda: eng.pagerank_precision(D, TOL), one / el.nV, (1 - D) * one / el.nV)]
        cases.append(cases[0])  # again, on the graph's kept tiles
        for s in seeds:
            e = np.eye(1, el.nV, s)[0]
            cases.append((lambda s=s: eng.ppr_precision(s, D, TOL), e, (1 - D) * e))
        for run, start, base in cases:
            ranks, st = run()
            assert np.abs(ranks.astype(np.float64) - reference(el, start, base)).sum() <= BOUND
            if hot is not None:
                assert st.kernel_launches == (4 if hot else 3) * st.iterations + 3


def rows(*lengths, nV=None, seed=1):
    """Vertex i has lengths[i] in-edges; the rest none."""
    rng = np.random.default_rng(seed)
    nV = nV or len(lengths) + 300
    dst = np.repeat(np.arange(len(lengths)), lengths)
    return EdgeList(nV, rng.integers(0, nV, len(dst)).astype(np.int32), dst.astype(np.int32))


@pytest.mark.parametrize("lengths", [
    (0,), (1,), (255,), (256,), (257,), (511, 1), (512,), (513, 0, 0, 7),
    (8, 8, 240, 256), (7, 1, 9, 239), (1,) * 256, (1,) * 257, (0, 1, 0, 2, 0, 3) * 100,
    (248, 16, 248), (20000,), (3, 20000, 5), (1, 300) * 40, (32, 33, 31) * 200,
], ids=str)
def test_row_lengths(lengths):
    check(rows(*lengths), hot=False, seeds=(0, len(lengths) + 299))


def test_few_edges_among_many_vertices():
    check(rows(5, 0, 300, nV=500_000), hot=False, seeds=(2, 499_999))


@pytest.mark.parametrize("graph,hot", [
    (lambda: EdgeList.rmat(18, 24, seed=3, symmetrize=False), False),  # too few edges
    (lambda: EdgeList.rmat(20, 12, seed=3, symmetrize=False), True),
    (lambda: rows(*[90] * 100_000, nV=200_000), False),  # no source stands out
    (lambda: rows(*[2800] * 3001, nV=20_000), True),  # a slot for every source
], ids=["few", "R-MAT", "even", "all hot"])
def test_hot_sources(graph, hot):
    check(graph(), hot=hot, seeds=(1,))
