"""Host logic (CPU, no GPU): rbk::simplify_queue (one-qubit gates merged, right
factors moved back through controls and CNOT targets) leaves the circuit's action
unchanged on random queues of every gate form (tests/host/simplify_check.cpp,
built with AddressSanitizer)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_simplified_queue_is_the_same_circuit(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "simplify_check"
    csrc = os.path.join(ROOT, "riken-braket_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-fno-omit-frame-pointer", "-I", csrc,
                    "-o", str(exe), os.path.join(ROOT, "tests", "host", "simplify_check.cpp"),
                    os.path.join(csrc, "rbk_plan.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr
    assert "ALL OK" in r.stdout
