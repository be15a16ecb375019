"""SSSP and CC as one persistent kernel (AUTO / LEARNED on small and medium
graphs): vertex data and iteration counts equal the multi-kernel push's and
the oracle's.  Out-degrees at the light / heavy entry limits (32, 128),
members without out-edges, more new members in a CTA than its stage holds,
dense iterations, odd and even iteration counts, capped and repeated runs."""
import numpy as np
import pytest

import oracle
from graphreduce_gb300 import GASEngineGPU, GasError
from graphreduce_gb300.engine import initial_vertex_data
from graphreduce_gb300.graph import EdgeList

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(libgas):
    return libgas


def degrees(nV, seed):
    rng = np.random.default_rng(seed)
    pairs = [rng.integers(0, nV, (2 * nV, 2))]
    for u, deg in enumerate((1, 31, 32, 33, 127, 128, 129, 256, 257, 5000)):
        if u < nV:
            pairs.append(np.stack([np.full(deg, u), rng.integers(0, nV, deg)], 1))
    e = np.concatenate(pairs).astype(np.int32)
    e = e[e[:, 0] % 7 != 6]  # vertices without out-edges
    w = rng.choice(np.array([0, 1, 5, 64, 100000], np.int32), len(e))
    return EdgeList(nV, e[:, 0].copy(), e[:, 1].copy(), w)


def star(leaves):
    """A hub, its leaves, and an edge from each leaf to the one after it."""
    i = np.arange(1, leaves + 1, dtype=np.int32)
    src = np.concatenate([np.zeros(leaves, np.int32), i[:-1]])
    dst = np.concatenate([i, i[1:]])
    w = np.concatenate([1 + i % 3, np.ones(leaves - 1, np.int32)]).astype(np.int32)
    return EdgeList(leaves + 1, src, dst, w)


def path(n):
    i = np.arange(n - 1, dtype=np.int32)
    return EdgeList(n, i, i + 1, np.ones(n - 1, np.int32))


GRAPHS = {
    "one vertex": lambda: EdgeList(1, np.zeros(1, np.int32), np.zeros(1, np.int32),
                                   np.zeros(1, np.int32)),
    "no edges": lambda: EdgeList(5000, *(np.zeros(0, np.int32),) * 3),
    "path of 38": lambda: path(38), "path of 39": lambda: path(39),
    "degrees 33": lambda: degrees(33, 1), "degrees 1025": lambda: degrees(1025, 2),
    "degrees 40001": lambda: degrees(40001, 3),
    "stage overflow": lambda: star(1_000_000),
    "dense iterations": lambda: EdgeList.rmat(17, 16, seed=9).with_uniform_weights(1, 64, 2),
    "islands": lambda: EdgeList.rmat(10, 8, seed=9).with_grid_islands(40, 32)
    .with_uniform_weights(1, 64, 2),
}


@pytest.mark.parametrize("name", GRAPHS)
@pytest.mark.parametrize("program", ["sssp", "cc"])
def test_one_kernel_equals_the_push_and_the_oracle(program, name):
    el = GRAPHS[name]()
    ref, rit = (oracle.sssp(el.nV, el.src, el.dst, el.weights, 0) if program == "sssp"
                else oracle.cc(el.nV, el.src, el.dst))
    eng = GASEngineGPU(program)
    init = initial_vertex_data(program, el.nV, 0)
    eng.setGraph(el.nV, init, el.nE, el.weights if program == "sssp" else None, el.src, el.dst)
    for schedule in ("auto", "push", "auto"):
        eng.upload_vertex_data(init)
        eng.setActive(0, el.nV)
        st = eng.run_schedule(schedule)
        out = np.empty(el.nV, np.int32)
        eng.download_vertex_data(out)
        np.testing.assert_array_equal(out, ref, err_msg=schedule)
        assert st.iterations == rit, schedule
        assert (st.kernel_launches == 1) == (schedule == "auto")
    # stopped after k iterations: the values are those of k pushes
    for cap in (1, 2):
        if rit <= cap:
            continue
        outs = []
        for schedule in ("auto", "push"):
            eng.upload_vertex_data(init)
            eng.setActive(0, el.nV)
            with pytest.raises(GasError) as err:
                eng.run_schedule(schedule, max_iterations=cap)
            assert err.value.status == 4
            out = np.empty(el.nV, np.int32)
            eng.download_vertex_data(out)
            outs.append(out)
        np.testing.assert_array_equal(outs[0], outs[1], err_msg=f"cap {cap}")
    eng.close()


@pytest.mark.parametrize("schedule,nV,one", [("auto", (1 << 22) - 1, True), ("auto", 1 << 22, False),
                                             ("learned", 1 << 20, True),
                                             ("learned", (1 << 20) + 1, False)])
def test_size_limits(schedule, nV, one):
    """At the largest sizes of the rule and just past them."""
    from graphreduce_gb300.learn import DATA, MLP
    rng = np.random.default_rng(5)
    src, dst = rng.integers(0, nV, (2, nV)).astype(np.int32)
    ref, rit = oracle.cc(nV, src, dst)
    eng = GASEngineGPU("cc")
    vd = initial_vertex_data("cc", nV)
    eng.setGraph(nV, vd, nV, None, src, dst)
    eng.set_schedule_model(MLP.load(DATA / "schedule_head.npz"))
    eng.setActive(0, nV)
    st = eng.run_schedule(schedule)
    eng.getResults()
    np.testing.assert_array_equal(vd, ref)
    assert st.iterations == rit and (st.kernel_launches == 1) == one
    eng.close()


@pytest.mark.parametrize("schedule,nV,one", [("auto", (1 << 22) - 1, True), ("auto", 1 << 22, False),
                                             ("learned", 1 << 21, True),
                                             ("learned", (1 << 21) + 1, False),
                                             ("learned", 5000, True)])
def test_sssp_size_limits(schedule, nV, one):
    """SSSP has a limit of its own under LEARNED."""
    from graphreduce_gb300.learn import DATA, MLP
    rng = np.random.default_rng(6)
    src, dst = rng.integers(0, nV, (2, 2 * nV)).astype(np.int32)
    w = rng.integers(1, 65, 2 * nV).astype(np.int32)
    s = int(src[0])
    ref, rit = oracle.sssp(nV, src, dst, w, s)
    eng = GASEngineGPU("sssp")
    vd = initial_vertex_data("sssp", nV, s)
    eng.setGraph(nV, vd, 2 * nV, w, src, dst)
    eng.set_schedule_model(MLP.load(DATA / "schedule_head.npz"))
    eng.setActive(0, nV)
    st = eng.run_schedule(schedule)
    eng.getResults()
    np.testing.assert_array_equal(vd, ref)
    assert st.iterations == rit and (st.kernel_launches == 1) == one
    eng.close()
