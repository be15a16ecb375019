"""Batched personalized PageRank on rows of several units: hubs over more units
than one group folds (16) and than a CTA has groups, rows ending exactly at a
unit's (128 in-edges) or a step's (8) end, an edge count that is no multiple of 8,
every vector width of the lanes, a graph without edges."""
import numpy as np
import pytest

import oracle
from graphreduce_gb300 import Batch
from graphreduce_gb300.graph import EdgeList
from test_batch_gpu import PPR_L1, PPR_TOL

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(libgas):
    return libgas


def rows(in_degrees, nV, seed):
    """Vertex v has in_degrees[v] in-edges (0 past the list) plus a ring."""
    rng = np.random.default_rng(seed)
    dst = np.concatenate([np.full(d, v) for v, d in enumerate(in_degrees)] + [np.arange(nV)])
    src = np.concatenate([rng.integers(0, nV, len(dst) - nV), (np.arange(nV) + 1) % nV])
    return EdgeList(nV, src.astype(np.int32), dst.astype(np.int32))


@pytest.fixture(scope="module")
def graphs():
    return [rows([7, 8, 9, 15, 63, 64, 65, 127, 128, 1, 2, 1100, 20000, 0, 50000], 3000, 1),
            EdgeList(5, np.zeros(0, np.int32), np.zeros(0, np.int32)),
            rows([63] * 40 + [64] * 40 + [5] * 3, 997, 2)]


@pytest.mark.parametrize("lanes", [1, 2, 3, 6, 16, 18])
@pytest.mark.parametrize("piece", [0, 8, 64, 1000])
def test_lanes_against_the_fp64_oracle(graphs, lanes, piece):
    b = Batch()
    for el in graphs:
        b.add_graph(el.nV, el.src, el.dst)
    b.build()
    rng = np.random.default_rng(lanes)
    seeds = np.stack([rng.integers(0, el.nV, lanes) for el in graphs]).astype(np.int32)
    seeds[0, 0] = 14   # the largest hub
    if lanes > 1:
        seeds[:, 1] = -1
    r = b.run(ppr_seeds=seeds, tol=PPR_TOL, piece_edges=piece)
    assert r.stats.ppr_residual <= PPR_TOL
    for g, el in enumerate(graphs):
        got = b.slice(r.rank, g)
        for l in range(lanes):
            if seeds[g, l] < 0:
                assert not got[:, l].any()
                continue
            ref, _, _ = oracle.ppr_fp64(el.nV, el.src, el.dst, int(seeds[g, l]), 0.85, 1e-13)
            assert np.abs(got[:, l].astype(np.float64) - ref).sum() <= PPR_L1, (g, l)
    b.close()
