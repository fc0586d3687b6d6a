"""The stand-alone GEMM harness (``tests/cuda``): it links the sources that the extension is built from, and its products agree with naive ones."""
import os
import shutil
import subprocess

import pytest

from mlx_sharding_b200.ops import build

CUDA = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cuda")


def test_harness_links(tmp_path):
    """A kernel file that the GEMM calls and the harness does not link is an undefined symbol here."""
    if not shutil.which(build._nvcc()):
        pytest.skip("no nvcc")
    subprocess.run(["bash", os.path.join(CUDA, "build.sh"), str(tmp_path)], check=True, capture_output=True, text=True)
    assert os.access(tmp_path / "gemm_test", os.X_OK) and os.access(tmp_path / "gemm_sweep", os.X_OK)


@pytest.mark.gpu
def test_harness_passes():
    exe = os.path.join(CUDA, "bin", "gemm_test")
    if not os.path.exists(exe):
        pytest.skip("tests/cuda/build.sh has not been run")
    r = subprocess.run([exe, "quick"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "PASSED" in r.stdout, r.stdout[-3000:]
