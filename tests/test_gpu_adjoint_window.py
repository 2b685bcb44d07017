"""The reverse flow kernel at the edges of its 26 x 27 window outputs and the
reverse sweep at the edges of its chunks, trees of 2 to 8 vertices in and out of
pre-order.  Data gradients equal the oracle's adjoint bit for bit, alpha
gradients (sums in another order) to 1e-9.  GPU only."""
import pytest

from tests.test_gpu_adjoint import assert_matches, problem, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(26, 27, 3), (27, 28, 5), (25, 26, 4), (53, 54, 2), (54, 55, 6), (2, 3, 2), (79, 29, 9)])
def test_window_edges(dims):
    w, truth = problem(41, dims, iterations=7)
    assert_matches(run_gpu(w, truth), run_oracle(w, truth), w, str(dims))


@pytest.mark.parametrize("parent", [[-1, 0], [-1, 0, 0], [-1, 0, 1, 1], [1, -1, 1, 0, 0], [-1, 0, 0, 1, 1, 2, 2],
                                    [-1, 0, 1, 1, 0, 4, 4], [-1, 0, 0, 0, 1, 1, 2, 2], [-1, 0, 0, 0, 0, 0, 0, 0],
                                    [3, 0, 0, -1, 3, 4, 4]])
@pytest.mark.parametrize("dims", [(8, 16, 1), (16, 16, 1), (33, 4, 2), (20, 13, 6)])
def test_sweep_chunks_and_trees(parent, dims):
    w, truth = problem(42, dims, parent, iterations=9, smooth_nodes=(len(parent) - 1,))
    assert_matches(run_gpu(w, truth), run_oracle(w, truth), w, str((parent, dims)))


@pytest.mark.parametrize("parent", [[1, -1], [2, 2, -1], [4, 4, 0, 0, -1], [5, 5, 0, 0, 1, -1], [6, 6, 0, 0, 1, 1, -1],
                                    [7, 7, 7, 0, 0, 1, 1, -1], [7, 7, 7, 7, 7, 7, 7, -1], [-1, 0, 1, 2, 3, 4]])
def test_sweep_with_the_root_last(parent):
    """The root's place among the staged arrays; a chain."""
    w, truth = problem(43, (20, 13, 6), parent, iterations=9, smooth_nodes=(0 if parent[0] >= 0 else 1,))
    assert_matches(run_gpu(w, truth), run_oracle(w, truth), w, str(parent))
