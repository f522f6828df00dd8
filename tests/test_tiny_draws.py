"""CPU check of the motion kernel's draws in float pairs (pair_math.h): no accepted
rounding differs from the double's, down to standard deviations of 1e-20 and normals
of 1e-23, and ordinary draws are still settled in pairs."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_draws_round_as_the_doubles(tmp_path):
    exe = tmp_path / "tiny_draws_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "tsdf_localization_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "tiny_draws_check.cpp"), "-o", str(exe), "-lm"], check=True)
    res = subprocess.run([str(exe), "3000000"], capture_output=True, text=True)
    print(res.stdout)
    assert res.returncode == 0, res.stdout
