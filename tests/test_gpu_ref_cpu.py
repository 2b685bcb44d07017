"""REF_CPU solves: CC that divides by multiplication and CC that does not,
iteration counts around where a label settles, ties between leaves and rows
whose last quad is partial.  Bit-identical to the oracle.  GPU only."""
import numpy as np
import pytest

from oracle import oracle as O
from robartsvtk_gb300 import REF_CPU, HMFSolver
from robartsvtk_gb300.synthetic import random_tree_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,parent", [((5, 3, 2), [-1, 0, 0]), ((33, 17, 6), [-1, 0, 1, 1, 0, 4, 4]),
                                         ((64, 9, 4), [-1, 0, 0, 0, 0])])
@pytest.mark.parametrize("cc", [0.25, 1.0, 0.3, 0.0078125, 0.9])
@pytest.mark.parametrize("iterations", [0, 1, 2, 3, 40])
def test_ref_cpu_matches_the_oracle(dims, parent, cc, iterations):
    w = random_tree_problem(17, dims, parent, iterations=iterations)
    rng = np.random.default_rng(17)
    for d in w.data.values():  # coarse values: many ties for the minimum, some exact zeros
        coarse = rng.random(d.shape) < 0.5
        d[coarse] = np.floor(d[coarse] * 2.0)
    with HMFSolver(w.dims, w.parent, REF_CPU) as s:
        for leaf, d in w.data.items():
            s.set_data(leaf, d)
        for v, a in w.alpha.items():
            s.set_smoothness_scalar(v, a)
        s.set_params(iterations, w.step, cc)
        s.solve()
        o = O.solve(w.dims, w.parent, w.data, w.smooth, w.alpha, iterations, w.step, cc, semantics=O.REF_CPU,
                    want_sink=True)
        for v in range(len(parent)):
            assert np.array_equal(s.sink(v), o["sink"][v].astype(np.float32)), v
            if parent[v] >= 0:
                assert np.array_equal(s.labels(v), o["u"][v].astype(np.float32)), v
