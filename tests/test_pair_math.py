"""CPU check of the float-pair trigonometry (pair_math.h): a rounding it accepts is
the double function's, rounded to float; the pairs lie within their stated bounds;
few roundings are left to the double functions."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_pairs_round_as_the_double_functions(tmp_path):
    exe = tmp_path / "pair_math_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "tsdf_localization_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "pair_math_check.cpp"), "-o", str(exe), "-lm"], check=True)
    res = subprocess.run([str(exe), "400000"], capture_output=True, text=True)
    print(res.stdout)
    assert res.returncode == 0, res.stdout
    rows = {r.split()[0]: r.split()[1:] for r in res.stdout.splitlines()}
    # stated bounds: angles 2^-42.5, normals 2^-42.5 of the 2^-41 they are rounded with
    for name in ("angles", "small", "large", "quarters", "log", "normals"):
        assert float(rows[name][2]) < -42.5
    # 2 x 2 roundings at 2^-41 of a float's 2^-24 to 2^-25: below 1 in 2,000
    for name in ("angles", "small", "large", "quarters"):
        assert int(rows[name][1]) < int(rows[name][0]) / 2000
