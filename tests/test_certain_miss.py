"""CPU check of certain_miss, by which the scoring kernels settle most points
outside the fast domain, against the oracle's getIndex."""
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_certain_miss_is_a_miss(tmp_path):
    exe = tmp_path / "miss_check"
    csrc = ROOT / "tsdf_localization_gb300" / "csrc"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = Path(nvcc).resolve().parent.parent / "include"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fopenmp", "-I", str(csrc), "-I",
                    str(ROOT / "include"), "-I", str(ROOT / "oracle"), "-I", str(inc),
                    str(ROOT / "tests" / "native" / "miss_check.cpp"), str(csrc / "map_build.cpp"), "-x", "c",
                    str(ROOT / "oracle" / "tsdf_oracle.c"), "-o", str(exe), "-lm"], check=True)
    res = subprocess.run([str(exe), "8000"], capture_output=True, text=True)
    print(res.stdout)
    assert res.returncode == 0, res.stdout
    f = dict(zip(res.stdout.split()[::2], res.stdout.split()[1::2]))
    # random points: well over half of the misses are settled
    assert int(f["settled"]) > 0.5 * int(f["misses"]) > 0
