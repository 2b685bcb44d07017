"""Data terms at the sizes where their kernel changes: double for small images, then
float-float with a voxel per thread, then with four; images of which some, none
or all voxels lie outside the float-float range, and warps that hold both.  The
Gaussian equals the restatement bit for bit; the logistic's library functions
may differ in the last bits of the double, which moves the float rounding of
about one value in 10^8 by an ulp (at most one of these in an array).  GPU only."""
import numpy as np
import pytest

from oracle import dataterm_oracle as DT
from robartsvtk_gb300 import data_term
from tests.test_gpu_term_paths import same

pytestmark = pytest.mark.gpu

SIZES = [16383, 16384, 16385, 32767, 32768, 32801, 40009, 262143, 262145, 524287, 524290]
IMAGES = {
    "inside": lambda r, n: r.normal(0.4, 0.2, n),
    "outside": lambda r, n: r.uniform(-1000, 1000, n),
    "some": lambda r, n: np.where(r.random(n) < 0.02, 4000.0, r.normal(0.4, 0.2, n)),
    "wide": lambda r, n: r.uniform(-1, 1, n) * np.exp2(r.uniform(-50, 50, n)),
}


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("image", sorted(IMAGES))
def test_sizes(n, image):
    torch = pytest.importorskip("torch")
    r = np.random.default_rng(n)
    x = IMAGES[image](r, n).astype(np.float32)
    y = r.normal(0.3, 0.4, n).astype(np.float32)
    dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    for op, k1 in ((DT.GAUSSIAN, 0.05), (DT.LOGISTIC, 3.0)):
        for entropy in (False, True):
            c = dict(k1=k1, c1=0.4, k2=2.0, c2=0.7, entropy=entropy)
            strict = op == DT.GAUSSIAN and entropy
            with np.errstate(all="ignore"):
                same(data_term(op, dx, **c).cpu().numpy(), DT.data_term(op, x, **c), strict)
                same(data_term(op, dx, dy, **c).cpu().numpy(), DT.data_term(op, x, y, **c), strict)
                if strict:
                    same(data_term(op, dx, normalize=True, **c).cpu().numpy(), DT.data_term(op, x, normalize=True, **c),
                         True)


@pytest.mark.parametrize("n", [1, 5, 1023, 1024, 70001])
@pytest.mark.parametrize("shift", [0, 1])
def test_constant_and_spike(n, shift):
    """One of two values; a spike constant that no float equals is never hit."""
    torch = pytest.importorskip("torch")
    x = np.random.default_rng(n).integers(0, 3, n + shift).astype(np.float32)
    x[-1] = np.float32(0.1)
    t = torch.from_numpy(x).cuda()[shift:]
    for op in (DT.CONSTANT, DT.SPIKE):
        for k1 in (1.0, 0.1, float(np.float32(0.1)), float("nan")):
            for entropy in (False, True):
                for normalize in (False, True):
                    c = dict(k1=k1, c1=0.25, c2=0.75, entropy=entropy, normalize=normalize)
                    same(data_term(op, t, **c).cpu().numpy(), DT.data_term(op, x[shift:], **c), True)
