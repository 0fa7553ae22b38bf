"""What a batch refuses: above 12 qubits (13 in complex<float>) instances take what
the engine's sweep takes, and are refused when the batch runs; at and below that size there
are no limits on exponents, strings and flip patterns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spec_and_terms(n, what):
    spec = [("H", (0,), None, 0.0, ()), ("EY", (1,), 0, -0.5, ())]
    terms = [("Z" * n, 1.0)]
    if what == "exponent":
        spec.append(("U", (0, 1), None, 0.0, (n + 1,)))
    elif what == "negative exponent":
        spec.append(("U", (0, 1), None, 0.0, (-(n + 1),)))
    elif what == "strings":
        terms = [("".join("Z" if (k >> b) & 1 else "I" for b in range(n)), 0.1) for k in range(129)]
    elif what == "flips":
        terms = [("".join("X" if (k >> b) & 1 else "I" for b in range(n)), 0.1) for k in range(65)]
    elif what == "character":
        terms.append(("Q" * n, 1.0))
    return spec, terms


@pytest.mark.parametrize("what", ["exponent", "negative exponent", "strings", "flips", "character"])
@pytest.mark.parametrize("precision,n", [(0, 13), (0, 15), (1, 14), (1, 15)])
def test_refused_when_the_batch_runs(pkg, precision, n, what):
    spec, terms = spec_and_terms(n, what)
    b = pkg.adjoint.Batch([(n, spec, 1, terms), (4, spec[:2], 1, [("ZIII", 1.0)])], precision=precision)
    with pytest.raises(pkg.RbkError) as e:
        b.run([np.zeros(1), np.zeros(1)])
    assert e.value.code == 1
    b.close()


@pytest.mark.parametrize("precision,n", [(0, 12), (1, 13)])
@pytest.mark.parametrize("what", ["exponent", "strings", "flips"])
def test_small_instances_have_no_such_limits(pkg, precision, n, what):
    spec, terms = spec_and_terms(n, what)
    b = pkg.adjoint.Batch([(n, spec, 1, terms)], precision=precision)
    energies, _ = b.run([np.zeros(1)])
    assert np.isfinite(energies).all()
    b.close()


@pytest.mark.parametrize("what", ["most exponent", "most strings", "most flips"])
@pytest.mark.parametrize("precision,n", [(0, 13), (1, 14)])
def test_the_limits_themselves_are_accepted(pkg, precision, n, what):
    spec, terms = spec_and_terms(n, what.split()[1])
    if what == "most exponent":
        spec[-1] = ("U", (0, 1), None, 0.0, (n,))
    else:
        terms = terms[:-1]
    b = pkg.adjoint.Batch([(n, spec, 1, terms)], precision=precision)
    energies, grads = b.run([np.full(1, 0.3)])
    e, g = pkg.adjoint.adjoint_gradient(n, spec, np.full(1, 0.3), terms)
    # 128 weights of 0.1 added up in another order: 12.8 * 128 roundings of 1.1e-16; in
    # complex<float> the amplitudes were rounded at up to 3 gates: 12.8 * 2 * 3 * 6e-8
    tol = 12.8 * (128 * 1.1e-16 if precision == 0 else 2 * 3 * 6e-8)
    assert abs(energies[0] - e) <= tol and np.abs(grads[0] - g).max() <= tol
    b.close()
