"""The flow kernel where its windows, pairs of columns and multiplier can go
wrong: volume edges around the 28 x 27 window outputs, odd widths, few planes,
and bounds alpha * S(x) from zero and denormals to far above any flow.  The
kernel evaluates the oracle's FP32 operations, so the result is the oracle's
bit for bit.  GPU only."""
import numpy as np
import pytest

from robartsvtk_gb300.synthetic import random_tree_problem
from tests.test_gpu_parity import assert_same, oracle, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(27, 26, 5), (28, 27, 4), (29, 28, 6), (55, 53, 3), (56, 54, 7), (57, 55, 2),
                                  (2, 2, 2), (3, 1, 4), (84, 30, 1), (85, 82, 9)])
@pytest.mark.parametrize("zchunk", [0, 3])
def test_window_edges(dims, zchunk):
    w = random_tree_problem(5, dims, [-1, 0, 0, 1, 1], iterations=9, smooth_nodes=(1, 3))
    assert_same(run_gpu(w, zchunk=zchunk), oracle(w), "%s zchunk %d" % (dims, zchunk))


@pytest.mark.parametrize("window", [32, 64])
def test_bounds_of_every_size(window):
    """Smoothness values spread over the exponents of float32, zeros and
    denormals among them: every branch of the projection multiplier."""
    w = random_tree_problem(8, (61, 70, 9), [-1, 0, 1, 1, 0], iterations=12, smooth_nodes=(1, 2, 3, 4))
    rng = np.random.default_rng(8)
    shape = w.dims[::-1]
    for v in w.smooth:
        s = np.exp2(rng.uniform(-140, 30, size=shape)).astype(np.float32)
        s[rng.random(shape) < 0.4] = np.float32(0.05)
        s[rng.random(shape) < 0.1] = np.float32(0.0)
        w.smooth[v] = s
    w.alpha[2] = 0.0
    assert_same(run_gpu(w, window=window), oracle(w), "bounds, %d rows" % window)
