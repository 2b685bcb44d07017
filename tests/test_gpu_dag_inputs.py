"""Graph solver: data terms on the device that lie elsewhere at the next solve
(the replayed iterations read the new ones).  GPU only."""
import numpy as np
import pytest

from robartsvtk_gb300 import DAGSolver
from tests.test_gpu_dag import DIAMOND, assert_exact, oracle_solve, random_dag
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_device_inputs_that_move():
    import torch
    w = random_dag(17, (24, 18, 12), 6, DIAMOND, iterations=7, smooth_nodes=(4,))
    w2 = random_dag(18, (24, 18, 12), 6, DIAMOND, iterations=7, smooth_nodes=(4,))
    w2.smooth, w2.alpha = w.smooth, w.alpha
    root = O.dag_forward(w.n, w.edges, w.weights)[0]
    keep = []
    with DAGSolver(w.dims, w.n, w.edges, w.weights) as s:
        for v, S in w.smooth.items():
            s.set_smoothness(v, S)
        for v, a in w.alpha.items():
            s.set_smoothness_scalar(v, a)
        s.set_params(w.iterations, w.step, w.cc)
        for p in (w, w2, w):
            for leaf, d in p.data.items():
                keep.append(torch.from_numpy(np.ascontiguousarray(d)).cuda())
                s.set_data(leaf, keep[-1])
            s.solve()
            got = {"u": {v: s.labels(v) for v in range(w.n) if v != root}, "sink": {v: s.sink(v) for v in range(w.n)}}
            assert_exact(got, oracle_solve(p), "moved inputs")
