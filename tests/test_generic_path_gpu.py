"""The general iteration (step API, run(), the generic schedule): expansion
by rows and row chunks, compaction with the next gather's tile partition.
Sizes at the edges of a bitmap word, a warp's run (512 vertices), a block
(4,096) and the largest count whose blocks sum their predecessors (2,048
blocks); out-degrees around the row / chunk limits (64, 256); in-degrees that
span gather tiles (2,048 items)."""
import numpy as np
import pytest

import oracle
from graphreduce_gb300 import GASEngineGPU, run_program
from graphreduce_gb300.engine import initial_vertex_data
from graphreduce_gb300.graph import EdgeList

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(libgas):
    return libgas


def graph(nV, seed):
    rng = np.random.default_rng(seed)
    pairs = [rng.integers(0, nV, (3 * nV if nV < 1 << 22 else nV // 8, 2))]
    for u, deg in enumerate((63, 64, 65, 255, 256, 257, 1000)):
        if deg < nV and u < nV:
            pairs.append(np.stack([np.full(deg, u), rng.integers(0, nV, deg)], 1))
    if nV > 40000:  # in-edges over many tiles, at and next to a hub
        for v, deg in ((7, 30000), (8, 2048), (nV - 1, 9000)):
            pairs.append(np.stack([rng.integers(0, nV, deg), np.full(deg, v)], 1))
    e = np.concatenate(pairs).astype(np.int32)
    return EdgeList(nV, e[:, 0].copy(), e[:, 1].copy(),
                    rng.integers(1, 65, len(e)).astype(np.int32))


@pytest.mark.parametrize("nV", [1, 2, 31, 32, 33, 511, 513, 4095, 4096, 4097, 50001,
                                2048 * 4096, 2048 * 4096 + 1])
def test_against_oracle(nV):
    el = graph(nV, nV)
    schedules = ("step", "generic") if nV < 1 << 22 else ("generic",)
    refs = {"bfs": oracle.bfs(nV, el.src, el.dst, 0), "cc": oracle.cc(nV, el.src, el.dst),
            "sssp": oracle.sssp(nV, el.src, el.dst, el.weights, 0)}
    for program, (ref, rit) in refs.items():
        for schedule in schedules:
            vd, it = run_program(program, el, 0, schedule)
            np.testing.assert_array_equal(vd, ref, err_msg=f"{program}/{schedule}")
            assert it == rit, (program, schedule)
    # run() from the host, then again from another active range
    eng = GASEngineGPU("cc")
    vd = initial_vertex_data("cc", nV)
    eng.setGraph(nV, vd, el.nE, None, el.src, el.dst)
    eng.setActive(0, nV)
    assert eng.run() == refs["cc"][1]
    eng.getResults()
    np.testing.assert_array_equal(vd, refs["cc"][0])
    eng.setActive(0, (nV + 1) // 2)  # converged: one iteration, nothing changes
    eng.run_schedule("generic")
    eng.getResults()
    np.testing.assert_array_equal(vd, refs["cc"][0])
    eng.close()


@pytest.mark.parametrize("nV", [33, 4097, 50001])
def test_pagerank_against_oracle(nV):
    el = graph(nV, nV + 1)
    rank, _ = oracle.pagerank(nV, el.src, el.dst)
    for schedule in ("step", "generic"):
        vd, _ = run_program("pagerank", el, 0, schedule)
        # another summation order over FP32 sums (n 2^-24 of the largest, about
        # 30,000 in-edges) and, where it crosses |delta| = 0.01, one more or
        # one fewer update of at most that size
        np.testing.assert_allclose(vd["rank"], rank, rtol=2e-3, atol=0.011)
