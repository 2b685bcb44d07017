"""How a single volume's iterations are launched on the default plan: whole
launches that overlap their successors while the flow step is resident at
once, the slab pipeline (in at least three slabs) from there on.  Both give
the oracle's results bit for bit, over odd and long iteration counts and with
the convergence log.  GPU only."""
import numpy as np
import pytest

from robartsvtk_gb300 import DAGSolver, HMFSolver
from robartsvtk_gb300.synthetic import random_tree_problem
from tests.test_gpu_batch import make_batch, solve_batch
from tests.test_gpu_dag import assert_exact, oracle_solve, random_dag
from tests.test_gpu_parity import assert_same, oracle, run_gpu

pytestmark = pytest.mark.gpu

FLAT3 = [-1, 0, 0, 0]
TREE8 = [-1, 0, 0, 1, 1, 2, 2, 3, 3, 4, 4, 5, 5, 6, 6]


@pytest.mark.parametrize("dims,parent,iterations,slabs", [
    ((64, 60, 48), FLAT3, 33, 1),         # one wave: 144 units
    ((61, 59, 47), FLAT3, 70, 1),         # odd axes, two long replays
    ((300, 9, 50), [-1, 0, 1, 1], 5, 1),  # windows in x only
    ((100, 80, 60), TREE8, 5, 3),         # 60 planes in thirds
    ((100, 80, 59), TREE8, 4, 3),         # the last slab shorter
    ((130, 120, 30), TREE8, 3, 2),        # too thin for thirds of 20 planes: two slabs of 15
    ((112, 112, 60), [-1, 0, 1, 1, 1, 0, 0], 2, 5),  # five slabs cost less than one wave
    ((168, 162, 62), [-1, 0, 0, 0, 0], 2, 1),        # one wave costs less than slabs
])
def test_default_plan(dims, parent, iterations, slabs):
    w = random_tree_problem(11, dims, parent, iterations=iterations, smooth_nodes=(1,))
    r = run_gpu(w)
    assert_same(r, oracle(w), str(dims))
    assert r["stats"]["launches"] == 1 + 2 * slabs * iterations


def test_whole_launches_with_the_log_and_continued():
    """The log's entries and the state after rounds of a continued solve are
    those of launches one by one (timing mode records no graphs)."""
    w = random_tree_problem(12, (60, 58, 52), FLAT3, iterations=0, smooth_nodes=(2,))
    out = []
    for timing in (False, True):
        with HMFSolver(w.dims, w.parent) as s:
            s.set_timing(timing)
            s.set_convergence_log(True)
            for leaf, d in w.data.items():
                s.set_data(leaf, d)
            for v, S in w.smooth.items():
                s.set_smoothness(v, S)
            for v, a in w.alpha.items():
                s.set_smoothness_scalar(v, a)
            logs = []
            for i, k in enumerate((35, 1, 4)):
                s.set_params(k, w.step, w.cc)
                s.solve() if i == 0 else s.solve_continue()
                logs.append(s.convergence())
            out.append((logs, [s.labels(v) for v in range(1, len(w.parent))], [s.sink(v) for v in range(len(w.parent))]))
    for a, b in zip(out[0][0], out[1][0]):
        assert len(a["max"]) and np.array_equal(a["max"], b["max"])
        np.testing.assert_allclose(a["mean"], b["mean"], rtol=1e-6)
    for a, b in zip(out[0][1] + out[0][2], out[1][1] + out[1][2]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dims,zchunk,iterations,slabs", [
    ((112, 112, 60), 0, 3, 5),   # the default plan's slabs
    ((30, 20, 24), 6, 35, 4),    # a long replay
    ((29, 21, 23), 5, 4, 5),     # odd axes, the last slab shorter
    ((29, 21, 23), 2, 4, 1),     # chunks too thin for slabs
    ((40, 30, 20), 0, 5, 1),     # one wave
])
def test_graph_in_slabs(dims, zchunk, iterations, slabs):
    """A graph's iterations; its last one runs fewer tasks, in whole launches.
    The second solve's inputs lie elsewhere."""
    import torch
    edges = [(0, 1), (1, 2), (1, 3), (0, 4), (4, 5), (4, 6), (4, 3)]
    w = random_dag(19, dims, 7, edges, iterations=iterations, smooth_nodes=(1, 4))
    o = oracle_solve(w)
    keep = []
    with DAGSolver(w.dims, w.n, w.edges, w.weights) as s:
        s.set_zchunk(zchunk)
        for v, S in w.smooth.items():
            s.set_smoothness(v, S)
        for v, a in w.alpha.items():
            s.set_smoothness_scalar(v, a)
        s.set_params(w.iterations, w.step, w.cc)
        for _ in range(2):
            for leaf, d in w.data.items():
                keep.append(torch.from_numpy(np.ascontiguousarray(d)).cuda())
                s.set_data(leaf, keep[-1])
            s.solve()
            assert_exact({"u": {v: s.labels(v) for v in range(1, w.n)}, "sink": {v: s.sink(v) for v in range(w.n)}}, o,
                         str(dims))
            assert s.stats()["launches"] == 1 + 2 * slabs * (iterations - 1) + 2


@pytest.mark.parametrize("dims", [
    [(40, 33, 100), (30, 41, 61), (57, 28, 35), (29, 27, 3)] * 3,  # one long chunk for some, several for others
    [(20, 18, 70), (9, 40, 33)],                                   # few windows: short chunks
])
def test_batch_default_plan(dims):
    ws = make_batch(21, dims, parent=[-1, 0, 0, 1, 1], iterations=3, smooth_nodes=(1,))
    got, _ = solve_batch(ws)
    for i, w in enumerate(ws):
        assert_same(got[i], oracle(w), "volume %d %s" % (i, w.dims))
