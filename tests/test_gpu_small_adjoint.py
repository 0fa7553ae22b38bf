"""Gradients of circuits that run in one launch -- single ones of up to 10 qubits
(one CTA) and batches of up to 15 (one CTA to 12, clusters of 2, 4 and 8 CTAs above) --
against the engine's sweep on the same circuits: every gate kind, parameters used
twice, SWAPs before and after rotations, fixed rotations, strings with Y and several
flips, and the sizes around each launch shape.

Tolerances: a gate rounds a state by some u = 4 * 1.1e-16 (complex<float>: 6e-8) of its
norm, so that count gates leave about u sqrt(count); 4 times that is allowed.  An energy
has it twice, times the weights of the strings; a parameter's overlap has it from both
states, forward and back, once for each gate that uses the parameter."""
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


def random_terms(pkg, n, rng):
    terms = [("".join(rng.choice(list("IXYZ"), n)), float(w)) for w in rng.standard_normal(9)]
    return terms + (pkg.circuits.ansatz_hamiltonian(n) if n > 2 else [])


def tolerances(precision, spec, params, terms):
    """Of the energy and of every parameter's derivative."""
    state = 4 * (4 * 1.1e-16 if precision == 0 else 6e-8) * np.sqrt(len(spec) + 1)
    weight = sum(abs(c) for _, c in terms)
    uses = np.zeros(params)
    for _, _, param, scale, _ in spec:
        if param is not None:
            uses[param] += abs(scale)
    return 2 * state * weight, 2 * uses * 4 * state * weight


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 9, 10, 11, 12, 13, 14, 15])
def test_one_launch_gradient_vs_engine_sweep(pkg, monkeypatch, precision, n):
    rng = np.random.default_rng(n)
    params = 7
    terms = random_terms(pkg, n, rng)
    ctx = pkg.adjoint.AdjointContext(n, precision)
    other = pkg.adjoint.AdjointContext(n)
    for count in (0, 1, 25, 300):
        spec = mixed_spec(n, rng, params, count)
        theta = rng.uniform(-3, 3, params)
        e, g = ctx.gradient(spec, theta, terms)
        monkeypatch.setenv("RBK_ADJOINT_PAIR_ROTATE", "0")
        e0, g0 = other.gradient(spec, theta, terms)
        monkeypatch.delenv("RBK_ADJOINT_PAIR_ROTATE")
        tol_e, tol_g = tolerances(precision, spec, params, terms)
        assert abs(e - e0) <= tol_e
        assert np.all(np.abs(g - g0) <= tol_g)
    ctx.close()
    other.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sizes", [(10, 1, 7, 10, 3), (11, 11), (12, 12, 12), (13, 13), (14, 14), (15, 15), (15, 13, 9, 14, 12, 11, 2)])
def test_batch_launch_vs_engine_sweep(pkg, monkeypatch, precision, sizes):
    """Circuits of 0, 1, 25 and 300 gates, several of one launch shape and of all of them in a batch."""
    rng = np.random.default_rng(100 * sum(sizes) + len(sizes))
    inst, thetas = [], []
    for n in sizes:
        for count in (300, 0, 25, 1):
            inst.append((n, mixed_spec(n, rng, 7, count), 7, random_terms(pkg, n, rng)))
            thetas.append(rng.uniform(-3, 3, 7))
    batch = pkg.adjoint.Batch(inst, precision=precision)
    monkeypatch.setenv("RBK_ADJOINT_PAIR_ROTATE", "0")
    contexts = {n: pkg.adjoint.AdjointContext(n) for n in sizes}
    for _ in range(2):  # the second run replays the graph with other parameters
        energies, grads = batch.run(thetas)
        for (n, spec, params, terms), theta, e, g in zip(inst, thetas, energies, grads):
            e0, g0 = contexts[n].gradient(spec, theta, terms)
            tol_e, tol_g = tolerances(precision, spec, params, terms)
            assert abs(e - e0) <= tol_e, (n, len(spec))
            assert np.all(np.abs(g - g0) <= tol_g), (n, len(spec))
        thetas = [t + 0.1 for t in thetas]
    batch.close()
    for ctx in contexts.values():
        ctx.close()


def test_invalid_circuits_are_still_refused(pkg):
    ctx = pkg.adjoint.AdjointContext(4)
    for bad in ([("H", (4,), None, 0.0, ())], [("CNOT", (1, 1), None, 0.0, ())], [("U", (0, 1), None, 0.0, (5,))]):
        with pytest.raises(pkg.RbkError):
            ctx.gradient(bad, np.zeros(1), [("ZIII", 1.0)])
    with pytest.raises(pkg.RbkError):
        ctx.gradient([], np.zeros(1), [("ZIIQ", 1.0)])
    ctx.close()
