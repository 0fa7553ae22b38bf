"""Straight passes (layers of uncontrolled 2x2 gates, runs of phase gates, and
CNOT / X gates that all fold into the exchanges): the planner's programs on the host against the gates one by
one, and the kernel against the oracle and against the general tile pass (tile
shape 0 has no straight form) at the smallest state of the kind, at odd sizes and
at every number of phases.  Tolerances: rounding 1e-16 (6e-8 in complex<float>) at
each of some 300 gates on amplitudes of 1 at most."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle
from conftest import ROOT


def test_straight_programs_are_exact(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "straight_check"
    csrc = os.path.join(ROOT, "riken-braket_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-fno-omit-frame-pointer", "-I", csrc,
                    "-o", str(exe), os.path.join(ROOT, "tests", "host", "straight_check.cpp"),
                    os.path.join(csrc, "rbk_plan.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr
    assert "ALL OK" in r.stdout


ANGLES = {"U3": 3, "U1": 1, "EZ": 1}


def cnot_circuit(n, rng, count, rare):
    ops = []
    for _ in range(count):
        a, b = (int(x) for x in rng.permutation(n)[:2])
        kind = str(rng.choice(["U3", "U3", "H", "X", "CNOT", "CNOT"] + rare))
        ops.append((kind, (a, b) if kind in ("CNOT", "CZ") else (a,), tuple(rng.uniform(-3, 3, ANGLES.get(kind, 0)))))
    return ops


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [13, 14, 16, 17])
def test_straight_passes_vs_oracle(pkg, precision, n):
    rng = np.random.default_rng(n)
    circuits = [pkg.circuits.brick(n, 5, seed=n), cnot_circuit(n, rng, 300, []), cnot_circuit(n, rng, 300, ["CZ", "U1", "Z", "EZ"]),
                pkg.circuits.ansatz(n, 4, seed=n)[0]]
    for ops in circuits:
        ref = oracle.COracle(n)
        ref.apply(ops)
        want = ref.amplitudes()
        # 1 .. 6 phases a pass, and more than a straight pass holds
        for budget in (1, 4, 8, 12, 16, 20, 30):
            got = {}
            for shape in (2, 0):
                s = pkg.State(n, precision)
                s.set_tile_shape(shape)
                s.set_pass_budget(budget)
                s.apply(ops)
                got[shape] = s.amplitudes()
            tol = 1e-13 if precision == 0 else 2e-5
            assert np.abs(got[2] - want).max() <= tol
            assert np.abs(got[2] - got[0]).max() <= tol
