"""The energy of a solver's labels (rows padded to a multiple of 4 floats) at the
edges of the march's tiles, 64 columns x 16 rows or 32 x 32 where rows are short:
odd widths, whose last pair is half a pair, ending at a tile's border and one
voxel to either side of it.  FP64 sums in another order: relative 1e-11.  GPU
only."""
import numpy as np
import pytest

from oracle import oracle as O
from robartsvtk_gb300 import HMFSolver
from robartsvtk_gb300.synthetic import random_tree_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(31, 33, 5), (32, 32, 4), (33, 31, 9), (63, 17, 5), (64, 16, 4), (65, 15, 6), (127, 17, 3),
                                  (129, 33, 2), (1, 31, 3)])
def test_energy_at_tile_edges(dims):
    parent = [-1, 0, 1, 1, 0]
    w = random_tree_problem(44, dims, parent, iterations=5, smooth_nodes=(1, 4))
    with HMFSolver(w.dims, w.parent) as s:
        for leaf, d in w.data.items():
            s.set_data(leaf, d)
        for v, S in w.smooth.items():
            s.set_smoothness(v, S)
        for v, a in w.alpha.items():
            s.set_smoothness_scalar(v, a)
        s.set_params(w.iterations, w.step, w.cc)
        s.solve()
        f0, f = s.energy()
        labels = {v: s.labels(v) for v in w.leaves}
    o = O.energy(w.dims, w.parent, w.data, labels, w.smooth)
    assert abs(f0 - o["f0"]) <= 1e-11 * abs(o["f0"])
    np.testing.assert_allclose(f, o["f"], rtol=1e-11, atol=1e-30)
