"""The general iteration's expansion by push and by pull: in-degrees around
the lane's 64 in-edges and the chunks of 256 after them, hits only at a row's
end, vertices without in-edges or out-edges, pulls that find nothing, and
frontiers on both sides of the direction rule.  Results and iteration counts
equal the oracle's."""
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


def weighted(nV, src, dst, seed=1):
    rng = np.random.default_rng(seed)
    return EdgeList(nV, np.asarray(src, np.int32), np.asarray(dst, np.int32),
                    rng.integers(1, 64, len(src)).astype(np.int32))


def in_degrees(*degs):
    """Vertex i of the first len(degs) has degs[i] in-edges from vertices that
    settle at once but for the last, whose values come down a path."""
    n, top = len(degs), max(degs) + 8
    src, dst = [], []
    for i, d in enumerate(degs):
        src += list(range(n, n + d - 1)) + [n + top]
        dst += [i] * d
    path = np.arange(n + top + 30, n + top, -1)
    return weighted(n + top + 31, src + list(path), dst + list(path - 1))


def random_rows(nV, seed):
    rng = np.random.default_rng(seed)
    src, dst = [rng.integers(0, nV, 2 * nV)], [rng.integers(0, nV, 2 * nV)]
    for u, d in enumerate((1, 31, 32, 33, 63, 64, 65, 319, 320, 321, 5000)):
        src += [rng.integers(0, nV, d), np.full(d, u % nV)]
        dst += [np.full(d, u % nV), rng.integers(0, nV, d)]
    src, dst = np.concatenate(src), np.concatenate(dst)
    keep = (src % 7 != 3) & (dst % 5 != 4)  # some without out-edges, some without in-edges
    return weighted(nV, src[keep], dst[keep])


GRAPHS = {
    "one edge": lambda: weighted(2, [0], [1]),
    "in-degrees": lambda: in_degrees(1, 2, 63, 64, 65, 66, 319, 320, 321, 322, 576, 577, 5000),
    "33 vertices": lambda: random_rows(33, 1),
    "1025 vertices": lambda: random_rows(1025, 2),
    "40001 vertices": lambda: random_rows(40001, 3),
    "misses": lambda: EdgeList.rmat(12, 16, seed=5).with_grid_islands(100, 20)
    .with_uniform_weights(1, 64, 3),
    "R-MAT": lambda: EdgeList.rmat(16, 16, seed=6).with_uniform_weights(1, 64, 3),
    "R-MAT directed": lambda: EdgeList.rmat(15, 20, seed=7, symmetrize=False)
    .with_uniform_weights(1, 64, 3),
}


@pytest.mark.parametrize("name", GRAPHS)
@pytest.mark.parametrize("program", ["bfs", "sssp", "cc"])
def test_generic_runs(program, name):
    el = GRAPHS[name]()
    with closing(GASEngineGPU(program)) as eng:
        for s in (0, el.nV - 1) if program != "cc" else (0, 0):
            ref, it = (oracle.bfs(el.nV, el.src, el.dst, s) if program == "bfs" else
                       oracle.sssp(el.nV, el.src, el.dst, el.weights, s) if program == "sssp" else
                       oracle.cc(el.nV, el.src, el.dst))
            vd = initial_vertex_data(program, el.nV, s if program == "sssp" else None)
            fresh = vd.copy()
            eng.setGraph(el.nV, vd, el.nE, el.weights if program == "sssp" else None,
                         el.src, el.dst)
            for _ in range(2):
                eng.upload_vertex_data(fresh)
                eng.setActive(*((s, s + 1) if program == "bfs" else (0, el.nV)))
                st = eng.run_schedule("generic", max_iterations=el.nV + 2)
                eng.getResults()
                np.testing.assert_array_equal(vd, ref)
                assert st.iterations == it


def test_neighbouring_hubs_of_many_chunks():
    """64 hubs that share two words of the next frontier, with 60 chunks of
    in-edges each, every third full of changed in-neighbours: warps set a word's
    bits while others test them to skip their chunk."""
    hubs, chunks, m = 64, 60, 3000
    rng = np.random.default_rng(8)
    s = hubs                     # the source, then m vertices it leads to, then m unreached
    reached, rest = s + 1 + np.arange(m), s + 1 + m + np.arange(m)
    row = [rng.choice(rest, 70)]
    for c in range(chunks):
        row.append(rng.choice(reached if c % 3 == 1 else rest, 256))
    row = np.concatenate(row)
    nV = s + 1 + 2 * m + 20
    path = np.concatenate([[5], np.arange(nV - 20, nV)])
    el = weighted(nV, np.concatenate([np.full(m, s), np.tile(row, hubs), path[:-1]]),
                  np.concatenate([reached, np.repeat(np.arange(hubs), len(row)), path[1:]]))
    ref, it = oracle.sssp(el.nV, el.src, el.dst, el.weights, s)
    assert (ref[:hubs] < 200).all()
    with closing(GASEngineGPU("sssp")) as eng:
        vd = initial_vertex_data("sssp", el.nV, s)
        fresh = vd.copy()
        eng.setGraph(el.nV, vd, el.nE, el.weights, el.src, el.dst)
        for _ in range(20):
            eng.upload_vertex_data(fresh)
            eng.setActive(0, el.nV)
            st = eng.run_schedule("generic", max_iterations=el.nV + 2)
            eng.getResults()
            np.testing.assert_array_equal(vd, ref)
            assert st.iterations == it
