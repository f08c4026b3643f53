"""The device loop's quotient by RAND_MAX (crand_unit: a reciprocal and one
residual step) equals the division, on the CPU."""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent


def test_crand_unit_is_the_division(tmp_path):
    exe = tmp_path / "crand_unit_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    str(HERE / "crand_unit_check.cpp"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "0\n"
