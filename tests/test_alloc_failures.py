"""Host logic (CPU, no GPU): a failure inside a call is reported by that call and
leaves the object usable.  tests/host/alloc_check.cpp runs rbk_capi.cpp over a fake CUDA
runtime that fails one allocation after the other.  Built with AddressSanitizer."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_calls_recover_from_failed_allocations(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "alloc_check"
    csrc = os.path.join(ROOT, "riken-braket_b200", "csrc")
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    # rbk_capi.cpp names launches that these calls never reach; only those they reach have a fake.
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-fno-omit-frame-pointer", "-no-pie",
                    "-Wl,--unresolved-symbols=ignore-in-object-files", "-I", csrc, "-I", os.path.join(ROOT, "include"),
                    "-I", cuda_inc, "-o", str(exe), os.path.join(ROOT, "tests", "host", "alloc_check.cpp"),
                    *(os.path.join(csrc, f) for f in ("rbk_capi.cpp", "rbk_plan.cpp", "rbk_rotate_plan.cpp"))], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert "ALL OK" in r.stdout


def test_failed_batch_runs_leave_no_work_in_flight(tmp_path):
    """tests/host/batch_check.cpp: rbk_batch.cu over fakes, the large instances' sweep failing."""
    if not shutil.which("g++"):
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "batch_check"
    csrc = os.path.join(ROOT, "riken-braket_b200", "csrc")
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-fno-omit-frame-pointer", "-I", csrc,
                    "-I", os.path.join(ROOT, "include"), "-I", cuda_inc, "-o", str(exe), "-x", "c++",
                    os.path.join(ROOT, "tests", "host", "batch_check.cpp"), os.path.join(csrc, "rbk_batch.cu")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert "ALL OK" in r.stdout
