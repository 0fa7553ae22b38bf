"""Host logic (CPU, no GPU): a C++ model of sample_scan_kernel
(tests/host/sample_scan_check.cpp, over the kernel's own rbk_sample_scan.h) gives
scanned values that never decrease and stay where a sum is zero.  Built with
AddressSanitizer."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_scanned_sums_never_decrease(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "sample_scan_check"
    csrc = os.path.join(ROOT, "riken-braket_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-fno-omit-frame-pointer", "-I", csrc,
                    "-o", str(exe), os.path.join(ROOT, "tests", "host", "sample_scan_check.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr
    assert "ALL OK" in r.stdout
