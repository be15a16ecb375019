"""Device CSR / CSC build at the edges of its tiles (8,192 keys) and passes
(8 bits), on edge lists in and out of either order, and the list of rows with
in-edges behind the dense pull."""
import numpy as np
import pytest

import oracle
from graphreduce_gb300 import GASEngineGPU, GasError
from graphreduce_gb300.engine import initial_vertex_data

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(libgas):
    return libgas


@pytest.mark.parametrize("order", ["unsorted", "by source", "by destination", "by both"])
@pytest.mark.parametrize("nV,nE", [(2, 1), (255, 8191), (256, 8192), (257, 8193), (70000, 40000),
                                   (4097, 100001), ((1 << 24) + 1, 70000)])
def test_orders(monkeypatch, nV, nE, order):
    monkeypatch.setenv("GAS_GRAPH_BUILD", "device")
    rng = np.random.default_rng(nV + nE)
    src, dst = rng.integers(0, nV, (2, nE)).astype(np.int32)
    if order == "by source":
        src.sort()
    elif order == "by destination":
        dst.sort()
    elif order == "by both":
        src.sort()
        dst.sort()
    w = rng.integers(0, 100001, nE).astype(np.int32)
    eng = GASEngineGPU("sssp")
    init = initial_vertex_data("sssp", nV, int(src[0]))
    eng.setGraph(nV, init, nE, w, src, dst)
    got = eng.graph_arrays()
    for off, out, wt, key, val in (("csr_off", "csr_dst", "csr_w", src, dst),
                                   ("csc_off", "csc_src", "csc_w", dst, src)):
        o, v, perm = oracle.edge_list_to_csr(nV, key, val)
        np.testing.assert_array_equal(got[off], o)
        np.testing.assert_array_equal(got[out], v)
        np.testing.assert_array_equal(got[wt], w[perm])
    if nV < 1 << 20:
        ref, it = oracle.sssp(nV, src, dst, w, int(src[0]))
        eng.setActive(0, nV)
        st = eng.run_schedule("pull")
        vd = np.empty(nV, np.int32)
        eng.download_vertex_data(vd)
        np.testing.assert_array_equal(vd, ref)
        assert st.iterations == it
    eng.close()


@pytest.mark.parametrize("nE", [5, 300001])
def test_bad_weight_is_named_and_leaves_the_graph(nE):
    nV = 1000
    rng = np.random.default_rng(nE)
    src, dst = rng.integers(0, nV, (2, nE)).astype(np.int32)
    w = np.full(nE, 100000, np.int32)
    eng = GASEngineGPU("sssp")
    init = initial_vertex_data("sssp", nV, 0)
    eng.setGraph(nV, init, nE, w, src, dst)
    for bad in (-1, 100001):
        v = w.copy()
        v[nE - 2] = v[nE - 1] = bad
        with pytest.raises(GasError, match=f"weight {bad} of edge {nE - 2} ") as err:
            eng.setGraph(nV, init, nE, v, src, dst)
        assert err.value.status == 1
    eng.setActive(0, nV)
    eng.run_schedule("auto")  # the first graph is still there
    eng.getResults()
    np.testing.assert_array_equal(init, oracle.sssp(nV, src, dst, w, 0)[0])
    eng.close()
