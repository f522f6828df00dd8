"""CPU check of the fixed-point scale of the likelihood sums (tsdfl_internal.h): as fine
as 62 bits allow whatever the form the kernels sum in, and the packed form only where
its values leave the hits' bits alone."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_scale_is_the_largest_that_fits(tmp_path):
    cuda = next((p for p in (Path("/usr/local/cuda/include"), Path("/usr/include")) if (p / "cuda_runtime.h").exists()),
                None)
    if cuda is None:
        pytest.skip("no CUDA headers")
    exe = tmp_path / "scale_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(cuda), "-I", str(ROOT / "include"), "-I",
                    str(ROOT / "tsdf_localization_gb300" / "csrc"), str(ROOT / "tests" / "native" / "scale_check.cpp"),
                    "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    print(res.stdout)
    assert res.returncode == 0, res.stdout
