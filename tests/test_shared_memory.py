"""The kernels' opt-in to more than 48 KB of shared memory belongs to a device: on a fake runtime of several
devices, and no kernel that keeps the record of it in another way."""
import re
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "replica_exchange_wang_landau_b200" / "csrc"


def test_opt_in_is_made_on_every_device(tmp_path):
    exe = tmp_path / "shared_memory_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I/usr/local/cuda/include",
                    str(ROOT / "tests" / "native" / "shared_memory_check.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout == "ok\n", res.stdout


def test_no_kernel_sets_the_attribute_by_itself():
    users = [p.name for p in sorted(CSRC.iterdir()) if re.search(r"\bcudaFuncSetAttribute\s*\(", p.read_text())]
    assert users == ["shared_memory.hpp"]
