"""The digit contraction (csrc/exact_gemm.cu) after a wait that gave up: the
check program links the library's objects and presets the status word that
such a wait would write, so that every later wait of the launch ends at once."""
import pathlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def check_output(tmp_path_factory):
    import build as B
    B.build()
    exe = tmp_path_factory.mktemp("status") / "exact_status_check"
    objs = [str(B.BUILD / f"{n}.o") for n in ("exact_gemm", "ff_ozaki")]
    r = subprocess.run([B.nvcc(), *B.ARCH, *B.NVCC_FLAGS, str(ROOT / "tests" / "csrc" / "exact_status_check.cu"), *objs,
                        "-o", str(exe), "-lcuda"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
    return run.stdout


def test_contraction_that_gives_up_returns(check_output):
    assert "0 bad" in check_output


def test_contraction_that_gives_up_raises_its_flag(check_output):
    """Its sums are then left to the FP64 kernels, also in the real-valued and
    half-sum forms, which report no status."""
    for slices in (6, 7):
        assert f"slices {slices}: flag 0, 1 with a set status, 0\n" in check_output
