"""The claims that the flow step's multiplier and the energy's root rest on: the
root corrected from the hardware's approximation is sqrtf's on every float of
its exponents, and the quotient formed from it the division's.  Both hang on the
device's approximation, so every value of the roots and four billion pairs of
the quotient are compared (tests/cpp/root_check.cu).  The data terms' float-float
forms against double arithmetic over 6 * 10^7 values: the Gaussian's equal; the
logistic's functions may round the last bits of the double otherwise, at most
one value in 10^7, by an ulp.  GPU only."""
import os
import subprocess

import pytest

from robartsvtk_gb300 import build, data_term
from robartsvtk_gb300.dataterm import GAUSSIAN, LOGISTIC

pytestmark = pytest.mark.gpu
SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp", "root_check.cu")


def test_roots_and_quotients_are_exact(tmp_path):
    exe = str(tmp_path / "root_check")
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", *build.ARCH, "-fmad=false", "-I", build.CSRC, "-o", exe, SRC],
                   check=True, capture_output=True)
    words = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert words[:6] == ["roots", "0", "energy", "0", "mults", "0"] and int(words[7]) > 3 << 30


@pytest.mark.parametrize("op,entropy,k,c", [
    (GAUSSIAN, True, 0.05, 0.4), (GAUSSIAN, True, 3.7, -12.3), (GAUSSIAN, True, 1e-3, 1e4),
    (LOGISTIC, True, 3.0, 0.4), (LOGISTIC, True, 12.0, 0.8), (LOGISTIC, False, 3.0, 0.4), (LOGISTIC, False, -40.0, 0.1)])
def test_terms_over_many_values(op, entropy, k, c):
    torch = pytest.importorskip("torch")
    n = 10_000_000
    g = torch.Generator(device="cuda")
    K, C = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (k, c))  # (a scalar divisor would multiply)
    for seed in range(6):
        g.manual_seed(seed)
        x = torch.randn(n, device="cuda", generator=g) * (0.5 if seed % 2 else 5.0 * abs(1.0 / k)) + c
        d = x.double()
        if op == GAUSSIAN:
            q = (d - C) / K
            want = 0.5 * q * q
        else:
            a = 1.0 + torch.exp(-(K * (d - C)))
            want = torch.log(a) if entropy else 1.0 / a
        got, want = data_term(op, x, k1=k, c1=c, entropy=entropy).view(torch.int32), want.float().view(torch.int32)
        off = (got - want).abs()
        assert int((off != 0).sum()) <= (0 if op == GAUSSIAN else 1) and int(off.max()) <= 1
