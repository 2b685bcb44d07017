"""The cell kernels that small volumes run (16 x 8 x 4 cells, trees of up to 8
vertices): cell edges, partial cells, one-voxel axes, every tree size, bounds
of every magnitude, odd iteration counts and continued solves.  Bit-identical
to the oracle and to the march.  GPU only."""
import numpy as np
import pytest

from robartsvtk_gb300 import HMFSolver
from robartsvtk_gb300.synthetic import random_tree_problem
from tests.test_gpu_parity import assert_same, oracle, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(16, 8, 4), (17, 9, 5), (15, 7, 3), (1, 1, 1), (1, 20, 1), (33, 1, 9), (40, 36, 28)])
@pytest.mark.parametrize("iterations", [1, 10])
def test_cell_edges(dims, iterations):
    w = random_tree_problem(3, dims, [-1, 0, 0, 1, 1], iterations=iterations, smooth_nodes=(1, 3))
    assert_same(run_gpu(w), oracle(w), str(dims))


@pytest.mark.parametrize("parent", [[-1, 0], [-1, 0, 0], [-1, 0, 1, 1], [-1, 0, 0, 0, 0], [-1, 0, 1, 2, 3, 3],
                                    [-1, 0, 1, 1, 0, 4, 4], [-1, 0, 0, 0, 1, 1, 2, 2], [1, -1, 1, 0, 0]])
def test_trees(parent):
    w = random_tree_problem(4, (21, 18, 9), parent, iterations=33, smooth_nodes=(len(parent) - 1,))
    assert_same(run_gpu(w), oracle(w), str(parent))


def test_bounds_of_every_size():
    w = random_tree_problem(8, (35, 19, 9), [-1, 0, 1, 1, 0], iterations=12, smooth_nodes=(1, 2, 3, 4))
    rng = np.random.default_rng(9)
    for v in w.smooth:
        s = np.exp2(rng.uniform(-140, 30, size=w.dims[::-1])).astype(np.float32)
        s[rng.random(s.shape) < 0.4] = np.float32(0.05)
        s[rng.random(s.shape) < 0.1] = np.float32(0.0)
        w.smooth[v] = s
    assert_same(run_gpu(w), oracle(w), "bounds")


def test_march_and_cells_continue_each_other():
    """Rounds of a continued solve on either path give the one long solve."""
    w = random_tree_problem(6, (37, 22, 13), [-1, 0, 0, 1, 1], iterations=0, smooth_nodes=(2,))
    ref = oracle(w, iterations=30)
    with HMFSolver(w.dims, w.parent) as s:
        for leaf, d in w.data.items():
            s.set_data(leaf, d)
        for v, S in w.smooth.items():
            s.set_smoothness(v, S)
        for v, a in w.alpha.items():
            s.set_smoothness_scalar(v, a)
        for k, zchunk in ((7, 0), (8, 4), (10, 0), (5, 3)):
            s.set_zchunk(zchunk)
            s.set_params(k, w.step, w.cc)
            s.solve() if k == 7 else s.solve_continue()
        for v in range(len(w.parent)):
            assert np.array_equal(s.sink(v), ref["sink"][v].astype(np.float32)), v
            if w.parent[v] >= 0:
                assert np.array_equal(s.labels(v), ref["u"][v].astype(np.float32)), v
