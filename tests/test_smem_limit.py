"""Shared-memory limits of kernels belong to a device and are asked for by several threads: the host-side class that keeps them,
built with g++, and its use by every launcher."""
import re
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "camelid_b200" / "csrc"


def test_limits_are_per_device_and_only_raised(tmp_path):
    exe = tmp_path / "smem_limit_host_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-o", str(exe), str(HERE / "smem_limit_host_check.cpp")], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr


def test_launchers_set_kernel_attributes_through_it():
    setters = [p.name for p in sorted(CSRC.iterdir()) if re.search(r"\bcudaFuncSetAttribute\b", p.read_text())] if CSRC.is_dir() else []
    assert setters == ["common.cuh"], setters
