"""Batched personalized PageRank on rows of several units: hubs over more units
than one group folds (16) and than a CTA has groups, rows ending exactly at a
unit's (128 in-edges) or a step's (8) end, an edge count that is no multiple of 8,
every vector width of the lanes, a graph without edges."""
import math

import numpy as np
import pytest

import oracle
from graphreduce_gb300 import Batch, GasError
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


def test_residual_has_the_bits_of_an_fp64_sum():
    """Steps of 2^-4, 2^-29 and 2^-54 in the rows of one thread: every partial
    sum fits 53 bits, so an FP64 sum of them is exact in any order, and 48 bits
    lose the smallest."""
    n = 100_000

    def fan(*degs):
        """A seed and a chain of vertices with degs[i] out-edges, all but one to
        a last vertex; the chain's end leads to n others as well."""
        k = len(degs)
        src, dst, sink = [], [], k + n
        for i, d in enumerate(degs):
            to = np.full(d, sink)
            if i < k - 1:
                to[0] = i + 1
            else:
                to[:n] = k + np.arange(n)
            src.append(np.full(d, i))
            dst.append(to)
        return EdgeList(sink + 1, np.concatenate(src).astype(np.int32),
                        np.concatenate(dst).astype(np.int32))
    i = np.arange(4, dtype=np.int32)
    graphs = [EdgeList(5, i, i + 1), fan(1, 1 << 4, 1 << 4, 1 << 17),
              fan(1, 1 << 16, 1 << 17, 1 << 17)]
    seeds = np.zeros((3, 32), np.int32)
    b = Batch()
    for el in graphs:
        b.add_graph(el.nV, el.src, el.dst)
    b.build()
    ranks = []
    for cap in (3, 4):
        r = np.empty((b.num_vertices, 32), np.float32)
        with pytest.raises(GasError):
            b.run(ppr_seeds=seeds, damping=0.5, tol=1e-30, max_ppr_iterations=cap, rank_out=r)
        assert (r == r[:, :1]).all()
        ranks.append(r[:, 0].astype(np.float64))
    step = np.abs(ranks[1] - ranks[0])
    assert {2.0 ** -4, 2.0 ** -29, 2.0 ** -54} <= set(step)
    want = math.fsum(step)
    assert want < 0.5 and (np.remainder(step * 2.0 ** 54, 1) == 0).all()
    assert math.fsum(step[step > 2.0 ** -54]) != want
    r = b.run(ppr_seeds=seeds, damping=0.5, tol=want)
    assert r.stats.ppr_iterations == 4
    assert list(r.stats.ppr_lane_residual[:32]) == [want] * 32
    b.close()


@pytest.mark.parametrize("lanes", [1, 2, 6, 16, 32])
def test_a_short_row_next_to_long_ones_is_summed_term_by_term(lanes):
    """A row with contributions c, c 2^-24 and c 2^-24, whose sum is a float but
    whose pairwise sum loses it; the hub's units are longer and share its walk."""
    p1, q1, p2, q2, v, sink, d = 1, 2, 3, 4, 5, 6, 1 << 12
    pairs = ([(0, p1), (0, q1), (p1, p2), (p2, v), (q1, q2)] + [(q1, sink)] * (d - 1)
             + [(q2, v)] * 2 + [(q2, sink)] * (d - 2))
    src, dst = np.array(pairs, np.int32).T
    b = Batch()
    b.add_graph(7, src.copy(), dst.copy())
    b.build()
    rank = np.empty((7, lanes), np.float32)
    with pytest.raises(GasError):
        b.run(ppr_seeds=np.zeros((1, lanes), np.int32), damping=0.5, tol=1e-30,
              max_ppr_iterations=3, rank_out=rank)
    assert (rank[v] == np.float32(2.0 ** -4 + 2.0 ** -27)).all()
    b.close()
