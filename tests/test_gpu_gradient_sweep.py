"""Gradients by the engine's sweep above the one-launch sizes: more rotations than
one round of kept partial sums holds (64 launches), and Hamiltonians that take each
form of the H psi kernel -- real and imaginary weights (even and odd numbers of Y),
terms without Z, neighbouring and distant ZZ pairs, signs over many qubits.
The energy is compared with the oracle's state, the gradient of single parameters
with the exact two-term shift rule on the energy.  complex<double> sums 2^13
products of rounding 1e-16 after some 200 gates; complex<float> rounds its states
to 6e-8 at every gate."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

N = 13


def hamiltonians(pkg):
    letters = lambda **at: "".join(at.get(f"q{i}", "I") for i in range(N))
    return {
        "x": [(letters(q0="X"), 0.7), (letters(q12="X", q5="X"), -0.4)],
        "y": [(letters(q1="Y"), 0.9), (letters(q2="Y", q9="Y"), 0.3), (letters(q3="Y", q4="X", q11="Z"), -0.6)],
        "zz": [(letters(**{f"q{a}": "Z", f"q{b}": "Z"}), 0.1 * (1 + a)) for a, b in ((0, 1), (2, 3), (0, 12), (4, 11), (6, 7))],
        "signs": [("Z" * N, 0.5), ("XZ" * 6 + "Y", -0.8), ("IZ" * 6 + "X", 1.1)],
        "all": pkg.circuits.ansatz_hamiltonian(N),
    }


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("form", ["x", "y", "zz", "signs", "all"])
def test_gradient_sweep(pkg, precision, form):
    terms = hamiltonians(pkg)[form]
    rng = np.random.default_rng(5)
    spec, params = [], 0
    for layer in range(6):
        for q in range(N):
            # single rotations between entanglers: many pair-rotate launches
            spec.append((str(rng.choice(["EX", "EY", "EZ"])), (q,), params, 0.5, ()))
            params += 1
            spec.append(("CNOT", (q, (q + 1 + layer) % N), None, 0.0, ()))
    theta = rng.uniform(-2, 2, params)
    ctx = pkg.adjoint.AdjointContext(N, precision)
    exact = pkg.adjoint.AdjointContext(N)
    e, g = ctx.gradient(spec, theta, terms)
    scale = 1 + sum(abs(c) for _, c in terms)
    tol = (1e-11 if precision == 0 else 1e-4) * scale
    for k in (0, 1, 30, 64, params - 1):
        shifted = []
        for s in (1, -1):
            t = theta.copy()
            t[k] += s * np.pi / 2  # e^{i theta/2 P}: period 2 pi
            shifted.append(exact.gradient(spec, t, terms)[0])
        assert abs(g[k] - 0.5 * (shifted[0] - shifted[1])) <= tol
    o = oracle.COracle(N)
    o.apply([(kind, q, () if param is None else (scale * theta[param],)) for kind, q, param, scale, _ in spec])
    assert abs(e - o.expectation(terms).real) <= tol
    ctx.close()
    exact.close()
