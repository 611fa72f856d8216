"""Digits of float-float factors (csrc/exact_gemm.cuh, ex_ff_digits) and the
error of the sums they enter."""
import pathlib
import subprocess

import numpy as np
import pytest

import workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu
ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_float_float_digits_are_exact_in_bf16(tmp_path):
    import build as B
    exe = tmp_path / "exact_digits_check"
    r = subprocess.run([B.nvcc(), *B.ARCH, *B.NVCC_FLAGS, str(ROOT / "tests" / "csrc" / "exact_digits_check.cu"), "-o",
                        str(exe), "-lcuda"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr


@pytest.mark.parametrize("case", [(24, 40, 1024), (64, 100, 3000)], ids=lambda c: "x".join(map(str, c)))
def test_band_sums_are_as_exact_as_float_float_terms(sigma_lib, case):
    """Normwise over the band values, averaged over eight fills: the float-float
    term kernels' own error is 7e-15 on these ranges."""
    nb, ng, nc = case
    err = []
    for seed in range(8):
        p = W.gpp_random(nb, 2, nc, ng, 700 + seed)
        o, g = O.gpp(p)[2], sigma_lib.gpp_host(p, sigma_lib.PREC_FP64)[2]
        err.append(np.linalg.norm(g - o) / np.linalg.norm(o))
    assert np.mean(err) <= 6.9e-15
