"""The division-free quotient and bin floor of the look-ahead sweep (csrc/common.cuh) against the
host's division, over millions of operands that include rounding boundaries and bin edges."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_division_routines_match_the_division(tmp_path):
    exe = tmp_path / "division_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I/usr/local/cuda/include",
                    str(ROOT / "tests" / "native" / "division_check.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.startswith("ok"), res.stdout
