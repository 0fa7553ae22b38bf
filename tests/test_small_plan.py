"""Host logic (CPU, no GPU): the one-CTA programs of small states planned by
rbk::plan_small, executed by a C++ model of small_circuit_kernel
(tests/host/small_check.cpp), equal the gates applied one by one, for every
size from 1 to 12 qubits, programs longer than one launch, SWAPs and layout maps
that are not the identity; and planning takes time linear in the queue where a
qubit is never a target.  The model is built with AddressSanitizer."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_small_programs_are_exact(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "small_check"
    csrc = os.path.join(ROOT, "riken-braket_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-fno-omit-frame-pointer", "-I", csrc,
                    "-o", str(exe), os.path.join(ROOT, "tests", "host", "small_check.cpp"),
                    os.path.join(csrc, "rbk_plan.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr
    assert "ALL OK" in r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("precision,n", [(p, n) for p in (0, 1) for n in (1, 2, 3, 6, 10, 11, 12, 13)])
def test_small_states_vs_oracle(pkg, precision, n):
    """Both sides of the small-state line (12 / 13 qubits), programs of one gate, of one launch and of several.
    complex<double>: 400 gates of rounding 2e-16 on amplitudes of at most 1; complex<float>: 400 roundings of 6e-8."""
    import oracle

    tol = 1e-12 if precision == 0 else 2e-5
    rng = np.random.default_rng(n)
    init = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    init /= np.linalg.norm(init)
    kinds = ["H", "X", "Y", "Z", "U1", "U2", "U3", "EX", "EY", "EZ"] if n == 1 else None
    for count in (1, 60, 400):
        ops = pkg.circuits.random_circuit(n, count, seed=10 * n + count, kinds=kinds)
        o = oracle.COracle(n)
        o.set_amplitudes(init)
        o.apply(ops)
        with pkg.State(n, precision) as s:
            s.upload(init)
            s.apply(ops)
            assert np.abs(s.spins() - o.spins()).max() <= tol
            assert np.abs(s.amplitudes().astype(np.complex128) - o.amplitudes()).max() <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("precision,n", [(p, n) for p in (0, 1) for n in (1, 2, 3, 4, 9, 10, 11, 12)])
def test_one_phase_programs_vs_oracle(pkg, precision, n):
    """One register phase of 1 to 9 gates: up to 8 run straight from HBM, 9 through shared memory.
    Targets on at most three qubits, controls and phases on any; tolerances as above."""
    import oracle

    tol = 1e-12 if precision == 0 else 2e-5
    rng = np.random.default_rng(50 + n)
    init = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    init /= np.linalg.norm(init)
    for count in (1, 2, 7, 8, 9):
        for _ in range(6):
            targets = [int(q) for q in rng.permutation(n)[:3]]
            ops = []
            for _ in range(count):
                t, c = targets[int(rng.integers(len(targets)))], int(rng.integers(n))
                x = [float(v) for v in rng.uniform(-3, 3, 3)]
                pick = int(rng.integers(9))
                ops.append([("U3", (t,), tuple(x)), ("H", (t,), ()), ("Y", (t,), ()), ("EY", (t,), (x[0],)), ("U1", (c,), (x[0],)),
                            ("Z", (c,), ()), ("EZ", (c,), (x[0],)), ("CNOT", (c, t), ()) if c != t else ("X", (t,), ()),
                            ("CZ", (c, t), ()) if c != t else ("X", (t,), ())][pick])
            o = oracle.COracle(n)
            o.set_amplitudes(init)
            o.apply(ops)
            with pkg.State(n, precision) as s:
                s.upload(init)
                s.apply(ops)
                assert np.abs(s.amplitudes().astype(np.complex128) - o.amplitudes()).max() <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 11, 12, 13])
def test_gates_launched_one_by_one_vs_oracle(pkg, n):
    import oracle

    ops = pkg.circuits.random_circuit(n, 60, seed=n)
    o = oracle.COracle(n)
    o.apply(ops)
    with pkg.State(n) as s:
        s.set_deferred(False)
        s.apply(ops)
        assert np.abs(s.amplitudes() - o.amplitudes()).max() <= 1e-12
