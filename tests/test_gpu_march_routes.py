"""The z-march (flow_tma_kernel, tree_bulk_n_kernel) on volumes small enough for
the cell kernels, by each of the ways a caller has of keeping it there: a window
of its own (the slab pipeline, a single slab among them), the kernels named in
the environment (whole launches that overlap), the pipeline switched off.
Single columns, rows and planes, window edges with the whole chunk marched, the
golden cases.  Bit-identical to the oracle; the reference's own kernels to
1e-4.  GPU only."""
import os

import numpy as np
import pytest

from robartsvtk_gb300 import HMFSolver
from robartsvtk_gb300.synthetic import random_tree_problem
from tests.golden.cases import CASES, problem
from tests.test_gpu_parity import GOLDEN, LABEL_TOL, assert_same, oracle

pytestmark = pytest.mark.gpu

TREE5, TREE7 = [-1, 0, 0, 1, 1], [-1, 0, 0, 1, 1, 2, 2]
ROUTES = ["window", "named", "off"]


def march(w, route, monkeypatch):
    if route == "named":
        monkeypatch.setenv("HMF_FLOW_KERNEL", "tma")
    with HMFSolver(w.dims, w.parent) as s:
        if route == "window":
            s.set_flow_window(32)
        if route == "off":
            s.set_pipeline(False)
        for leaf, d in w.data.items():
            s.set_data(leaf, d)
        for v, S in w.smooth.items():
            s.set_smoothness(v, S)
        for v, a in w.alpha.items():
            s.set_smoothness_scalar(v, a)
        s.set_params(w.iterations, w.step, w.cc)
        s.solve()
        assert s.pipeline == (route == "window" and s.zchunk() >= 3)
        slabs = -(-w.dims[2] // s.zchunk()) if s.pipeline else 1
        assert s.stats()["launches"] == 1 + 2 * slabs * w.iterations
        n = len(w.parent)
        u = np.zeros((n,) + w.dims[::-1], np.float32)
        sink = np.zeros_like(u)
        for v in range(n):
            sink[v] = s.sink(v)
            if w.parent[v] >= 0:
                u[v] = s.labels(v)
        return {"u": u, "sink": sink}


@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("dims,parent,smooth_nodes,iterations", [
    ((5, 4, 3), [-1, 0, 0, 0], (), 7),
    ((1, 1, 1), [-1, 0], (), 3),
    ((1, 1, 9), [-1, 0, 0], (), 12),
    ((1, 1, 400), [-1, 0, 0], (1,), 5),     # a single column in many chunks
    ((40, 1, 1), [-1, 0, 0], (1,), 12),
    ((1, 40, 1), [-1, 0, 0], (1,), 12),
    ((31, 17, 1), [-1, 0, 0, 0], (2,), 15),
    ((64, 16, 40), TREE7, (1, 2, 3, 4, 5, 6), 9),
    ((70, 19, 23), [-1, 0, 1, 2, 2, 1, 0], (3, 4), 11),
    ((20, 12, 6), [-1, 0, 0], (), 4),
    ((24, 16, 9), [-1, 0, 0, 0], (), 33),
])
def test_shapes(dims, parent, smooth_nodes, iterations, route, monkeypatch):
    w = random_tree_problem(21, dims, parent, iterations=iterations, smooth_nodes=smooth_nodes)
    assert_same(march(w, route, monkeypatch), oracle(w), "%s %s" % (route, dims))


@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("dims", [(27, 26, 5), (28, 27, 4), (29, 28, 6), (55, 53, 3), (56, 54, 7), (57, 55, 2),
                                  (2, 2, 2), (3, 1, 4), (84, 30, 1), (85, 82, 9)])
def test_window_edges(dims, route, monkeypatch):
    w = random_tree_problem(5, dims, TREE5, iterations=9, smooth_nodes=(1, 3))
    assert_same(march(w, route, monkeypatch), oracle(w), "%s %s" % (route, dims))


@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("name", sorted(CASES))
def test_golden_cases(name, route, monkeypatch):
    w = problem(name)
    r = march(w, route, monkeypatch)
    assert_same(r, oracle(w), name)
    golden = os.path.join(GOLDEN, "ref_cuda_golden.npz")
    if os.path.exists(golden):  # vectors of the reference's own CUDA kernels
        assert np.abs(r["u"] - np.load(golden)[name + "/u"]).max() <= LABEL_TOL
