"""Every FP64 host call where the device has no room, or only some, for the
exact contractions' workspaces: same results, and no call refused that its
inputs and partial sums fit; and every form with an operand outside the
contractions' range, which gives the FP64 kernels' bits.  Free memory is simulated (csrc/no_room_check.cu,
linked with the library's objects); with too little of it the calls take the
gated copies of the GPP drop-in and each form's FP64 kernels."""
import pathlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_host_calls_with_little_memory(tmp_path):
    import build as B
    B.build()
    exe = tmp_path / "no_room_check"
    wrap = [x for n in ("cudaMalloc", "cudaFree", "cudaMemGetInfo") for x in ("-Xlinker", f"--wrap={n}")]
    r = subprocess.run([B.nvcc(), *B.ARCH, *B.NVCC_FLAGS, str(ROOT / "tests" / "csrc" / "no_room_check.cu"),
                        *[str(B.BUILD / (s.stem + ".o")) for s in B.sources()], "-o", str(exe), *wrap, "-lcuda"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=280)
    assert run.returncode == 0 and "\n0 bad" in run.stdout, run.stdout + run.stderr
