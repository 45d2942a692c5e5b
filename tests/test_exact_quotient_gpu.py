"""The exact kernels' branch-free reciprocals and quotients against IEEE
division, on the device (exact_quotient_check.cu)."""
import shutil
import subprocess
from pathlib import Path

import pytest

from hicar_b200 import build

pytestmark = pytest.mark.gpu
HERE = Path(__file__).resolve().parent


def test_quotients_equal_ieee_division(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    exe = tmp_path / "exact_quotient_check"
    flags = [f for f in build.NVCC_FLAGS if f not in ("-Xptxas", "-v")]
    subprocess.run([nvcc, *flags, str(HERE / "exact_quotient_check.cu"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and res.stdout.count("mismatches=0") == 4, res.stdout
