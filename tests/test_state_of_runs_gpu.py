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


class Filled:
    """All of the device's memory taken but for about `leave` bytes."""

    def __init__(self, leave):
        import torch
        torch.cuda.empty_cache()
        self.taken = []
        for step in (1 << 33, 1 << 30, 1 << 26, 1 << 23):
            while torch.cuda.mem_get_info()[0] > leave + step:
                self.taken.append(torch.empty(step, dtype=torch.uint8, device="cuda"))

    def release(self):
        import torch
        self.taken.clear()
        torch.cuda.empty_cache()


def test_batch_runs_after_one_that_found_no_memory():
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
            full = Filled(128 << 20)  # 32 lanes' rows take 256 MB
            with pytest.raises(GasError):
                b.run(**{f"{kind}_sources": many})
            full.release()
            r = b.run(**{f"{kind}_sources": one})
            got = r.depth if kind == "bfs" else r.dist
            reached = depth >= 0
            np.testing.assert_array_equal(got[reached, 0], depth[reached])
            r = b.run(**{f"{kind}_sources": many})
            got = r.depth if kind == "bfs" else r.dist
            np.testing.assert_array_equal(got[reached], np.repeat(depth[reached][:, None], 32, 1))
