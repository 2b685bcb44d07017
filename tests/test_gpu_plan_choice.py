"""Which kernels and launches a solve takes, and what the calls that choose them
promise: settings that the caller made stay in force, the pipeline's getter says
how the next solve runs, and a failed autotune changes nothing.  Results are the
oracle's bit for bit on every route.  GPU only."""
import os
import subprocess
import sys

import numpy as np
import pytest

from robartsvtk_gb300 import DAGSolver, HMFError, HMFSolver
from robartsvtk_gb300.synthetic import random_tree_problem
from tests.test_gpu_parity import oracle

pytestmark = pytest.mark.gpu

TREE5 = [-1, 0, 0, 1, 1]
TREE15 = [-1, 0, 0, 1, 1, 2, 2, 3, 3, 4, 4, 5, 5, 6, 6]
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def fill(s, w):
    for leaf, d in w.data.items():
        s.set_data(leaf, d)
    for v, S in w.smooth.items():
        s.set_smoothness(v, S)
    for v, a in w.alpha.items():
        s.set_smoothness_scalar(v, a)
    s.set_params(w.iterations, w.step, w.cc)


def assert_oracle(s, w, what=""):
    ref = oracle(w)
    for v in range(len(w.parent)):
        assert np.array_equal(s.sink(v), ref["sink"][v].astype(np.float32)), (what, v)
        if w.parent[v] >= 0:
            assert np.array_equal(s.labels(v), ref["u"][v].astype(np.float32)), (what, v)


@pytest.mark.parametrize("dims", [(40, 36, 28), (90, 75, 33)])
def test_failed_autotune_leaves_the_plan(dims):
    w = random_tree_problem(27, dims, TREE5, iterations=7, smooth_nodes=(1,))
    with HMFSolver(w.dims, w.parent) as s:
        s.set_flow_window(64)
        s.set_zchunk(5)
        s.set_flow_units(2)
        with pytest.raises(HMFError, match="[Mm]issing data"):
            s.autotune()
        assert (s.flow_window, s.zchunk(), s.flow_units) == (64, 5, 2)
        fill(s, w)
        s.solve()
        assert_oracle(s, w, dims)


@pytest.mark.parametrize("calls", [
    [("zchunk", 5), ("units", 0)],
    [("zchunk", 5), ("units", 4), ("units", 0)],
    [("units", 2), ("zchunk", 5), ("zchunk", 0)],
    [("window", 64), ("units", 0)],
    [("window", 64), ("zchunk", 0)],
    [("window", 32), ("zchunk", 5), ("zchunk", 0)],
])
def test_a_setting_stays_until_it_is_set_to_zero(calls):
    """A plan of the caller's is pipelined at any size, whatever other setting
    is restored after it; with every setting restored the default plan runs."""
    w = random_tree_problem(28, (40, 30, 60), TREE5, iterations=6, smooth_nodes=(1,))  # default chunks of 3 planes or more
    with HMFSolver(w.dims, w.parent) as s:
        setters = {"zchunk": s.set_zchunk, "units": s.set_flow_units, "window": s.set_flow_window}
        for name, value in calls:
            setters[name](value)
        fill(s, w)
        s.solve()
        slabs = -(-w.dims[2] // s.zchunk())
        assert slabs > 1 and s.stats()["launches"] == 1 + 2 * slabs * w.iterations
        assert_oracle(s, w, calls)
        for name in ("window", "zchunk", "units"):
            setters[name](0)
        s.solve()
        assert s.stats()["launches"] == 1 + 2 * w.iterations
        assert_oracle(s, w, calls)


def test_a_window_restores_the_default_chunk():
    with HMFSolver((40, 30, 20), TREE5) as s:
        z = s.zchunk()
        s.set_zchunk(5)
        s.set_flow_window(0)
        w = random_tree_problem(28, (40, 30, 20), TREE5, iterations=6)
        fill(s, w)
        s.solve()
        assert s.zchunk() == z and s.stats()["launches"] == 1 + 2 * w.iterations


TUNED = """
import sys
from robartsvtk_gb300 import HMFSolver
from robartsvtk_gb300.synthetic import random_tree_problem
from tests.test_gpu_plan_choice import TREE5, assert_oracle, fill
w = random_tree_problem(30, (40, 36, 28), TREE5, iterations=9, smooth_nodes=(1,))
with HMFSolver(w.dims, w.parent) as s:
    fill(s, w)
    if "tune" in sys.argv:
        s.autotune()
    s.solve()
    assert_oracle(s, w)
    print("plan", s.flow_window, s.zchunk(), s.flow_units)
"""


def tuned_process(cache, *args):
    """The plan of a context in a process of its own, which reads `cache`."""
    env = dict(os.environ, HMF_AUTOTUNE_CACHE=str(cache))
    r = subprocess.run([sys.executable, "-c", TUNED, *args], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return [int(x) for x in r.stdout.split("plan")[1].split()]


def test_autotune_of_a_small_volume(tmp_path):
    """The small volume's own kernels are a candidate, and its plans are cached
    apart from plans that were not timed against them."""
    cache = tmp_path / "tuned"
    default = tuned_process(cache)
    plan = tuned_process(cache, "tune")
    key, *saved = cache.read_text().split()
    assert key.startswith("cells/") and tuned_process(cache) == plan
    if int(saved[2]) == 0:
        assert plan == default
    cache.write_text("%s 16 5 2\n" % key)
    assert tuned_process(cache) == [64, 5, 2]
    cache.write_text("%s 8 7 0\n" % key)  # the small volume's kernels won: the default plan
    assert tuned_process(cache) == default
    cache.write_text("%s 16 5 2\n" % key[len("cells/"):])  # tuned without them
    assert tuned_process(cache) == default


@pytest.mark.parametrize("dims,parent,default", [((40, 30, 60), TREE5, False), ((64, 60, 48), TREE5, False),
                                                 ((100, 80, 60), TREE15, True)])
def test_the_pipeline_getter_says_how_the_next_solve_runs(dims, parent, default):
    """A small volume's own kernels, one wave in whole launches, and slabs."""
    w = random_tree_problem(31, dims, parent, iterations=5, smooth_nodes=(1,))
    with HMFSolver(w.dims, w.parent) as s:
        fill(s, w)
        slabs = -(-dims[2] // s.zchunk())
        for switch, expected in ((None, default), (True, default), (False, False), (True, default)):
            if switch is not None:
                s.set_pipeline(switch)
            assert s.pipeline == expected, switch
            s.solve()
            assert s.stats()["launches"] == 1 + 2 * (slabs if expected else 1) * w.iterations
            assert_oracle(s, w, (dims, switch))


def test_the_pipeline_getter_of_graphs():
    edges = [(0, 1), (1, 2), (1, 3), (0, 4), (4, 5), (4, 6), (4, 3)]
    for dims, more, pipelined in (((40, 30, 20), [], False), ((200, 200, 90), [], True),
                                  ((200, 200, 90), [(4, 3)], False)):  # a repeated edge: the general sweep
        with DAGSolver(dims, 7, edges + more) as s:
            assert s.pipeline == pipelined
            s.set_pipeline(False)
            assert not s.pipeline


@pytest.mark.parametrize("dims,cells", [((40, 36, 28), True), ((24, 20, 16), True), ((8, 8, 300), True),
                                        ((64, 16, 60), True), ((300, 280, 1), False), ((200, 200, 1), False),
                                        ((1, 9000, 1), False), ((52, 52, 32), False)])
def test_small_volumes_by_their_cells(dims, cells, tmp_path):
    """Whether a volume's own kernels are its default (the autotuner's key says
    so) goes by whole and partial 16 x 8 x 4 cells, not by voxels: flat and
    narrow volumes march.  On a GPU of 152 SMs, to which the line belongs."""
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("another number of SMs: another line")
    code = TUNED.replace("(40, 36, 28)", str(dims))
    env = dict(os.environ, HMF_AUTOTUNE_CACHE=str(tmp_path / "tuned"))
    r = subprocess.run([sys.executable, "-c", code, "tune"], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert (tmp_path / "tuned").read_text().startswith("cells/") == cells


@pytest.mark.parametrize("dims,parent", [((8, 8, 6000), [-1, 0, 0, 0]), ((5, 30, 4700), [-1, 0, 0])])
def test_a_long_thin_volume_is_not_cut_into_many_slabs(dims, parent):
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("another number of SMs: another plan")
    w = random_tree_problem(33, dims, parent, iterations=3)
    with HMFSolver(w.dims, w.parent) as s:
        fill(s, w)
        s.solve()
        assert not s.pipeline and s.stats()["launches"] == 1 + 2 * w.iterations
        assert_oracle(s, w, dims)
