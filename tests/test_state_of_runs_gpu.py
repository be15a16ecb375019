"""What runs keep between calls: state made on the run's own stream, state
after a run that found no memory, and the memory that set_graph and build take
before any run asks for it."""
from contextlib import closing

import numpy as np
import pytest

import oracle
from graphreduce_gb300 import Batch, GASEngineGPU, GasError
from graphreduce_gb300.engine import initial_vertex_data
from graphreduce_gb300.graph import EdgeList

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(libgas):
    return libgas


@pytest.fixture
def busy_default_stream():
    """The default stream at work for some 200 ms; what is put on it waits."""
    import torch

    def start():
        torch.cuda._sleep(400_000_000)
    yield start
    torch.cuda.synchronize()


def test_first_batch_run_on_a_stream_of_its_own(busy_default_stream):
    import torch
    el = EdgeList.rmat(12, 16, seed=3)
    srcs = np.array([[0, 5, 9, 77]], np.int32)
    for rep in range(3):
        s = torch.cuda.Stream()
        with closing(Batch()) as b:
            b.add_graph(el.nV, el.src, el.dst)
            b.build(stream=s)
            if rep:  # (the first one loads the kernels)
                busy_default_stream()
            r = b.run(bfs_sources=srcs, stream=s)
            # the default stream is still busy: the run did not use it
            assert rep == 0 or not torch.cuda.default_stream().query()
        for l, v in enumerate(srcs[0]):
            ref, _ = oracle.bfs(el.nV, el.src, el.dst, int(v))
            np.testing.assert_array_equal(r.depth[:, l], ref)
        torch.cuda.synchronize()


@pytest.mark.parametrize("program", ["bfs", "cc"])
def test_first_loop_run_on_a_stream_of_its_own(program, busy_default_stream):
    import torch
    el = EdgeList.rmat(12, 16, seed=3)
    ref, it = (oracle.bfs(el.nV, el.src, el.dst, 5) if program == "bfs"
               else oracle.cc(el.nV, el.src, el.dst))
    for rep in range(3):
        s = torch.cuda.Stream()
        with closing(GASEngineGPU(program)) as eng:
            vd = initial_vertex_data(program, el.nV)
            eng.setGraph(el.nV, vd, el.nE, None, el.src, el.dst, stream=s)
            eng.setActive(*((5, 6) if program == "bfs" else (0, el.nV)), stream=s)
            if rep:
                busy_default_stream()
            st = eng.run_schedule("push", stream=s)
            assert rep == 0 or not torch.cuda.default_stream().query()
            eng.getResults(stream=s)
        np.testing.assert_array_equal(vd, ref)
        assert st.iterations == it
        torch.cuda.synchronize()


@pytest.fixture
def fill():
    """fill(leave): all of the device's memory but for about `leave` bytes is
    taken; fill(None): none is."""
    import torch
    taken = []

    def to(leave):
        taken.clear()
        torch.cuda.empty_cache()
        for step in (1 << 33, 1 << 30, 1 << 26, 1 << 23) if leave is not None else ():
            while torch.cuda.mem_get_info()[0] > leave + step:
                taken.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
    yield to
    to(None)


def test_batch_runs_after_one_that_found_no_memory(fill):
    """The lanes' rows do not fit: the run fails, and a later run of the lanes
    that ran before makes its rows anew."""
    n = 1 << 21
    i = np.arange(n - 1, dtype=np.int32)
    i = i[i % 1000 != 999]
    with closing(Batch()) as b:
        b.add_graph(n, i, i + 1, np.ones(len(i), np.int32))
        b.build()
        depth = np.arange(n) % 1000
        depth[1000:] = -1
        one = np.zeros((1, 1), np.int32)
        many = np.zeros((1, 32), np.int32)
        for kind in ("bfs", "sssp"):
            b.run(**{f"{kind}_sources": one})
            fill(128 << 20)  # 32 lanes' rows take 256 MB
            with pytest.raises(GasError):
                b.run(**{f"{kind}_sources": many})
            fill(None)
            r = b.run(**{f"{kind}_sources": one})
            got = r.depth if kind == "bfs" else r.dist
            reached = depth >= 0
            np.testing.assert_array_equal(got[reached, 0], depth[reached])
            r = b.run(**{f"{kind}_sources": many})
            got = r.depth if kind == "bfs" else r.dist
            np.testing.assert_array_equal(got[reached], np.repeat(depth[reached][:, None], 32, 1))


def drop_of(f):
    """(result, bytes of device memory that f() takes)"""
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    r = f()
    torch.cuda.synchronize()
    return r, before - torch.cuda.mem_get_info()[0]


def chain(nV):
    """Every vertex 1000 k leads along a path to 1000 k + 999."""
    i = np.arange(nV - 1, dtype=np.int32)
    i = i[i % 1000 != 999]
    return EdgeList(nV, i, i + 1)


def test_set_graph_leaves_the_memory_of_runs_that_nobody_asked_for(fill):
    """The one-kernel BFS's buffers (32 V + E bytes) come with set_graph where
    they are at most a quarter of the free memory, and are given back to the
    multi-kernel loop where that finds no memory."""
    nV = 1 << 22
    el = chain(nV)
    size = 2 * (nV + el.nE // 32 + 1) * 16
    vd = initial_vertex_data("bfs", nV)
    fresh = vd.copy()
    ref = np.full(nV, -1, np.int32)
    ref[:1000] = np.arange(1000)

    def run(eng, schedule):
        eng.upload_vertex_data(fresh)
        eng.setActive(0, 1)
        st = eng.run_schedule(schedule)
        eng.getResults()
        np.testing.assert_array_equal(vd, ref)
        return st

    def graph():
        eng = GASEngineGPU("bfs")
        eng.setGraph(nV, vd, el.nE, None, el.src, el.dst)
        return eng
    with closing(graph()) as eng:
        run(eng, "auto")  # (kernels are loaded)
    eng, ample = drop_of(graph)
    eng.close()
    fill(ample - size + 3 * size)  # what the graph takes, and 3 times the buffers
    eng, tight = drop_of(graph)
    assert ample - tight > 0.9 * size
    with closing(eng):
        assert run(eng, "auto").kernel_launches == 1  # they fit all the same
        fill(None)
        fill(48 << 20)  # not enough for the loop's 20 V
        assert run(eng, "push").kernel_launches > 1
        fill(None)
        assert run(eng, "auto").kernel_launches == 1


def test_build_leaves_the_memory_of_traversals_to_ppr(fill):
    """The frontier of the batch's traversals: not with build where it is more
    than a quarter of the free memory, and given back to a PPR run."""
    nV = 1 << 22
    el = chain(nV)
    size = 16 * nV

    def build():
        b = Batch()
        b.add_graph(nV, el.src, el.dst)
        b.build()
        return b
    seeds = np.zeros((1, 4), np.int32)
    b, _ = drop_of(build)
    ref, need = drop_of(lambda: b.run(ppr_seeds=seeds, tol=1e-3).rank)
    b.close()
    b, ample = drop_of(build)
    with closing(b):
        fill(32 << 20)
        with pytest.raises(GasError):  # the plan does not fit
            b.run(ppr_seeds=seeds, tol=1e-3)
        fill(None)
        assert (b.run(bfs_sources=seeds).depth[:1000, 0] == np.arange(1000)).all()
    b = build()
    with closing(b):
        fill(need - size // 2)
        np.testing.assert_array_equal(b.run(ppr_seeds=seeds, tol=1e-3).rank, ref)
        fill(None)
        r = b.run(bfs_sources=seeds)  # makes its frontier again
        assert (r.depth[:1000, 0] == np.arange(1000)).all()
    fill(ample - size + 3 * size)
    b, tight = drop_of(build)
    fill(None)
    assert ample - tight > 0.9 * size
    with closing(b):
        np.testing.assert_array_equal(b.run(ppr_seeds=seeds, tol=1e-3).rank, ref)
