"""The systematic resampler's block counters: a call leaves them at zero whatever they
held, so calls that overlapped on one context spoil no later call."""
import shutil
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


def test_every_call_leaves_the_counters_at_zero(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    lib_dir = ROOT / "tsdf_localization_gb300" / "_lib"
    exe = tmp_path / "resample_counters_check"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O1", "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "tsdf_localization_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "resample_counters_check.cu"), "-o", str(exe),
                    "-L", str(lib_dir), "-ltsdfl", "-Xlinker", f"-rpath={lib_dir}"], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    print(res.stdout, res.stderr)
    assert res.returncode == 0, res.stdout + res.stderr
