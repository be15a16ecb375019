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
