"""BFS as one persistent kernel: depths and iteration counts equal the
oracle's and the multi-kernel loop's.  Out-degrees at the limits of queue
entries (32, 128), in-degrees at those of a thread's and a warp's scan (29,
128), more new vertices in a CTA than its stage holds, top-down levels whose
finds are not queued followed by ones that need the queue, ranges of sources,
vertices visited before the run, and the largest graph that takes the kernel."""
import os
from contextlib import closing

import numpy as np
import pytest

import oracle
from graphreduce_gb300 import GASEngineGPU
from graphreduce_gb300.engine import initial_vertex_data
from graphreduce_gb300.graph import EdgeList

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(libgas):
    return libgas


def edges(nV, *pairs):
    e = np.concatenate([np.stack(np.broadcast_arrays(np.atleast_1d(a), b), 1)
                        for a, b in pairs])
    return EdgeList(nV, e[:, 0].astype(np.int32), e[:, 1].astype(np.int32))


def degrees(nV, seed, reverse):
    rng = np.random.default_rng(seed)
    pairs = [(rng.integers(0, nV, 2 * nV), rng.integers(0, nV, 2 * nV))]
    for u, d in enumerate((1, 28, 29, 30, 31, 32, 33, 127, 128, 129, 157, 158, 285, 5000)):
        pairs.append((np.full(d, u % nV), rng.integers(0, nV, d)))
    return edges(nV, *(p[::-1] if reverse else p for p in pairs))


def late_hit(nV):
    """Vertex nV-1 has in-edges from every vertex; only the last of them, in
    CSC order, is near the source."""
    i = np.arange(nV - 1)
    return edges(nV, (i, nV - 1), (nV - 2, nV - 1), (i[:-1] + 1, i[:-1]))


def star_and_path(leaves, tail):
    """A hub, its leaves, and a path out of the last one: a level of all the
    leaves between levels of one vertex."""
    i = np.arange(1, leaves + 1)
    t = np.arange(leaves, leaves + tail)
    return edges(leaves + tail + 1, (0, i), (t, t + 1))


def big_then_small(n):
    """Each of n vertices of level 1 leads to three of level 2, which share
    one successor, the head of a path."""
    a = np.arange(1, n + 1)
    b = n + 1 + np.arange(3 * n)
    t = 4 * n + 1 + np.arange(50)
    return edges(4 * n + 52, (0, a), (np.repeat(a, 3), b), (b, 4 * n + 1), (t, t + 1))


GRAPHS = {
    "one vertex": lambda: edges(1, (0, 0)),
    "33 vertices": lambda: degrees(33, 1, False),
    "out-degrees": lambda: degrees(40001, 3, False),
    "in-degrees": lambda: degrees(40001, 3, True),
    "late hit 29": lambda: late_hit(30), "late hit 30": lambda: late_hit(31),
    "late hit 158": lambda: late_hit(159), "late hit 9000": lambda: late_hit(9001),
    "stage overflow": lambda: star_and_path(1_000_000, 40),
    "not queued, then queued": lambda: big_then_small(300_000),
    "R-MAT": lambda: EdgeList.rmat(18, 16, seed=5),
    "R-MAT directed": lambda: EdgeList.rmat(19, 8, seed=6, symmetrize=False),
}


def runs(el, schedule, ranges, one_kernel, visited=()):
    before = os.environ.get("GAS_BFS_SMALL")
    os.environ["GAS_BFS_SMALL"] = "1" if one_kernel else "0"
    out = []
    try:
        with closing(GASEngineGPU("bfs")) as eng:
            vd = initial_vertex_data("bfs", el.nV)
            vd[list(visited)] = 7
            fresh = vd.copy()
            eng.setGraph(el.nV, vd, el.nE, None, el.src, el.dst)
            for a, b in ranges:
                eng.upload_vertex_data(fresh)
                eng.setActive(a, b)
                st = eng.run_schedule(schedule, max_iterations=el.nV + 2)
                eng.getResults()
                out.append((vd.copy(), st))
    finally:
        if before is None:
            del os.environ["GAS_BFS_SMALL"]
        else:
            os.environ["GAS_BFS_SMALL"] = before
    return out


@pytest.mark.parametrize("schedule", ["auto", "pull"])
@pytest.mark.parametrize("name", GRAPHS)
def test_depths_and_counts(name, schedule):
    el = GRAPHS[name]()
    ranges = [(0, 1), (el.nV // 2, el.nV // 2 + 1), (0, min(el.nV, 40)), (0, el.nV),
              (max(0, el.nV - 2), max(1, el.nV - 1)), (0, 1)]
    if schedule == "pull" and name in ("stage overflow", "not queued, then queued"):
        ranges = ranges[:2]
    got = runs(el, schedule, ranges, True)
    want = runs(el, schedule, ranges, False)
    for (a, b), (vd, st), (wvd, wst) in zip(ranges, got, want):
        np.testing.assert_array_equal(vd, wvd)
        assert st.iterations == wst.iterations
        assert st.kernel_launches == 1 < wst.kernel_launches
        if b == a + 1:
            ref, it = oracle.bfs(el.nV, el.src, el.dst, a)
            np.testing.assert_array_equal(vd, ref)
            assert st.iterations == it


def test_vertices_visited_before_the_run_stay():
    el = EdgeList.rmat(14, 8, seed=8)
    hub, _ = el.max_out_degree_vertex()
    visited = [v for v in range(0, el.nV, 3) if v != hub]
    got = runs(el, "auto", [(hub, hub + 1), (0, 50)], True, visited)
    want = runs(el, "auto", [(hub, hub + 1), (0, 50)], False, visited)
    for (vd, st), (wvd, wst) in zip(got, want):
        np.testing.assert_array_equal(vd, wvd)
        assert (vd[visited] == 7).all() and st.iterations == wst.iterations


@pytest.mark.parametrize("nV,one_kernel", [(1 << 23, True), ((1 << 23) + 1, False)])
def test_largest_graph(nV, one_kernel):
    rng = np.random.default_rng(4)
    hops = np.sort(rng.choice(nV, 60, replace=False))
    hops[-1] = nV - 1
    el = edges(nV, (hops[:-1], hops[1:]), (hops[30], rng.integers(0, nV, 100_000)))
    (vd, st), = runs(el, "auto", [(int(hops[0]), int(hops[0]) + 1)], True)
    ref, it = oracle.bfs(el.nV, el.src, el.dst, int(hops[0]))
    np.testing.assert_array_equal(vd, ref)
    assert st.iterations == it and (st.kernel_launches == 1) == one_kernel


def test_records_on_larger_graphs():
    """Tracing and profiling on a graph of more than 2^18 vertices: records
    and launches per iteration."""
    el = EdgeList.rmat(19, 8, seed=2)
    s, _ = el.max_out_degree_vertex()
    ref, it = oracle.bfs(el.nV, el.src, el.dst, s)
    with closing(GASEngineGPU("bfs")) as eng:
        vd = initial_vertex_data("bfs", el.nV)
        fresh = vd.copy()
        eng.setGraph(el.nV, vd, el.nE, None, el.src, el.dst)
        eng.setActive(s, s + 1)
        assert eng.run_schedule("auto").kernel_launches == 1
        for switch in (eng.set_trace, eng.set_profiling):
            switch(True)
            eng.upload_vertex_data(fresh)
            eng.setActive(s, s + 1)
            st = eng.run_schedule("auto")
            eng.getResults()
            np.testing.assert_array_equal(vd, ref)
            assert st.iterations == it and st.kernel_launches > 1
            if switch == eng.set_trace:
                assert len(eng.trace()) == it
            else:
                p = eng.profile()
                assert p.push_launches + p.pull_launches > 1
            switch(False)


def test_wide_levels_in_a_row():
    """26 top-down levels one after the other whose finds are only marked
    (320 K out-edges each, more than two per thread of the grid), so that each
    level makes its queue from the bitmap right after one that did: the makes'
    counts must not be cleared while the next one adds to them.  Run often, as
    a lost count shows by timing only."""
    rng = np.random.default_rng(11)
    layers, n = 40, 20_000
    u = np.arange(n * (layers - 1))
    src = np.repeat(u, 16)
    dst = (src // n + 1) * n + rng.integers(0, n, len(src))
    dst[::16] = u + n             # every vertex of the next layer is found
    dst[1::16 * n] = dst[::16 * n]
    hubs = np.arange(0, len(src), 16 * n)  # vertex 0 of a layer: rows of several entries
    for h in hubs:
        src[h + 16:h + 16 * 20] = src[h]
    order = np.argsort(src, kind="stable")
    el = EdgeList(n * layers, src[order].astype(np.int32), dst[order].astype(np.int32))
    want = np.repeat(np.arange(layers, dtype=np.int32), n)
    got = runs(el, "auto", [(0, n)] * 40, True)
    for vd, st in got:
        np.testing.assert_array_equal(vd, want)
        assert (st.iterations, st.push_iters, st.pull_iters) == (layers, 26, 13)
        assert st.kernel_launches == 1
