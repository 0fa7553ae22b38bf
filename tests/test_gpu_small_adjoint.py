"""Gradients of circuits that run in one launch (up to 15 qubits: one CTA to 12,
clusters of 2, 4 and 8 CTAs above) against the engine's sweep on the same
circuits: every gate kind, parameters used twice, SWAPs before and after
rotations, fixed rotations, and the sizes around each launch shape.
complex<double>: both sum 2^15 products of rounding 1e-16 after some 300 gates;
complex<float>: the engine rounds its states to 6e-8 at every gate."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mixed_spec(n, rng, params, count):
    one = ["H", "X", "Y", "Z", "U1", "U2", "U3", "EX", "EY", "EZ"]
    two = ["CNOT", "CZ", "U", "SWAP"]
    spec = []
    for _ in range(count):
        kind = str(rng.choice(one + (two if n > 1 else []) + ["EX", "EY", "EZ"] * 3))
        q = tuple(int(x) for x in rng.permutation(n)[:2 if kind in two else 1])
        param, scale, angles = None, 0.0, tuple(float(x) for x in rng.uniform(-2, 2, 3))
        if kind in ("EX", "EY", "EZ") and rng.random() < 0.8:
            param, scale = int(rng.integers(params)), float(rng.choice([-0.5, 0.5, 1.25]))
        if kind == "U":
            angles = (float(rng.integers(1, n + 1) * rng.choice([-1, 1])),)
        spec.append((kind, q, param, scale, angles))
    return spec


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 9, 10, 11, 12, 13, 14, 15])
def test_one_launch_gradient_vs_engine_sweep(pkg, monkeypatch, precision, n):
    rng = np.random.default_rng(n)
    params = 7
    terms = [("".join(rng.choice(list("IXYZ"), n)), float(w)) for w in rng.standard_normal(9)]
    terms += pkg.circuits.ansatz_hamiltonian(n) if n > 2 else []
    ctx = pkg.adjoint.AdjointContext(n, precision)
    other = pkg.adjoint.AdjointContext(n)
    for count in (0, 1, 25, 300):
        spec = mixed_spec(n, rng, params, count)
        theta = rng.uniform(-3, 3, params)
        e, g = ctx.gradient(spec, theta, terms)
        monkeypatch.setenv("RBK_ADJOINT_PAIR_ROTATE", "0")
        e0, g0 = other.gradient(spec, theta, terms)
        monkeypatch.delenv("RBK_ADJOINT_PAIR_ROTATE")
        tol = (1e-11 if precision == 0 else 1e-3) * (1 + np.abs(g0).max() + sum(abs(c) for _, c in terms))
        assert abs(e - e0) <= tol
        assert np.abs(g - g0).max() <= tol
    ctx.close()
    other.close()


def test_invalid_circuits_are_still_refused(pkg):
    ctx = pkg.adjoint.AdjointContext(4)
    for bad in ([("H", (4,), None, 0.0, ())], [("CNOT", (1, 1), None, 0.0, ())], [("U", (0, 1), None, 0.0, (5,))]):
        with pytest.raises(pkg.RbkError):
            ctx.gradient(bad, np.zeros(1), [("ZIII", 1.0)])
    with pytest.raises(pkg.RbkError):
        ctx.gradient([], np.zeros(1), [("ZIIQ", 1.0)])
    ctx.close()
