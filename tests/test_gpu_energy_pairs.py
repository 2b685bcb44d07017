"""The energy of images of even width, two voxels per thread: widths and tile
edges, trees of 1 to 8 vertices, against the oracle.  FP64 sums in another
order: relative 1e-11.  GPU only."""
import numpy as np
import pytest

from oracle import oracle as O
from robartsvtk_gb300 import decomposition_energy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 1, 1), (3, 5, 4), (32, 33, 5), (34, 16, 9), (64, 31, 3), (66, 17, 13), (130, 3, 2)])
@pytest.mark.parametrize("parent", [[-1, 0], [-1, 0, 0, 0], [-1, 0, 1, 1, 0], [-1, 0, 1, 2, 2, 1, 0],
                                    [-1, 0, 0, 1, 1, 2, 2, 0, 0]])
def test_energy_of_pairs(dims, parent):
    r = np.random.default_rng(5)
    shape = dims[::-1]
    leaves = [v for v in range(1, len(parent)) if v not in parent]
    lab = {v: np.where(r.random(shape) < 0.3, 0.0, r.random(shape)).astype(np.float32) for v in leaves}
    dat = {v: r.random(shape).astype(np.float32) for v in leaves}
    sm = {len(parent) - 1: r.random(shape).astype(np.float32)}
    o = O.energy(dims, parent, dat, lab, sm)
    f0, f = decomposition_energy(dims, parent, dat, lab, sm)
    assert abs(f0 - o["f0"]) <= 1e-11 * abs(o["f0"])
    np.testing.assert_allclose(f, o["f"], rtol=1e-11, atol=1e-30)
