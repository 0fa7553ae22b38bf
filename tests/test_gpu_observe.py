"""One-qubit and diagonal observables in tiled reads of the whole state: sizes
below, at and above the 2^11-amplitude tile, more diagonal strings than one
launch holds (64), strings of one weight and of many, X / Y strings on every
qubit, and strings that take the general read (several flips, complex weights on
diagonals), against numpy in FP64.  The sums of 2^n terms are formed in FP64 on both
sides: 1e-13 times the sum of |coefficients| bounds both roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pauli_value(a, s):
    """<a| P |a> for the string s (character k on qubit k)."""
    b, n = a, len(s)
    for q, c in enumerate(s):
        if c == "I":
            continue
        v = b.reshape(1 << (n - 1 - q), 2, 1 << q)
        m = {"X": [[0, 1], [1, 0]], "Y": [[0, -1j], [1j, 0]], "Z": [[1, 0], [0, -1]]}[c]
        b = np.stack([m[0][0] * v[:, 0] + m[0][1] * v[:, 1], m[1][0] * v[:, 0] + m[1][1] * v[:, 1]], axis=1).reshape(-1)
    return np.vdot(a, b)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 5, 10, 11, 12, 14, 19, 20])
def test_expectation_and_spins_vs_numpy(pkg, precision, n):
    rng = np.random.default_rng(n)
    a = (rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)) * (1 + np.arange(1 << n) % 7)
    a = (a / np.linalg.norm(a)).astype(np.complex128 if precision == 0 else np.complex64)
    wide = a.astype(np.complex128)
    one = lambda c, q: "".join(c if k == q else "I" for k in range(n))  # noqa: E731
    terms = [(one("X", q), rng.standard_normal() + 1j * rng.standard_normal()) for q in range(n)]
    terms += [(one("Y", q), 0.5) for q in range(0, n, 2)]
    terms += [("".join(rng.choice(list("IZ"), n)), w) for w in rng.choice([1.0, -0.25, 3.0], 20)]
    terms += [("".join(rng.choice(list("IZ"), n)), float(w)) for w in rng.standard_normal(55)]
    terms += [("".join(rng.choice(list("IXYZ"), n)), 0.3) for _ in range(3)] + [("Z" * n, 0.2 + 0.1j)]
    with pkg.State(n, precision) as s:
        s.upload(a)
        if n > 1:
            s.swap(0, n - 1)  # a layout map that is not the identity
            wide = np.swapaxes(wide.reshape([2] * n), 0, n - 1).reshape(-1)
        want = sum(c * pauli_value(wide, t) for t, c in terms)
        scale = sum(abs(c) for _, c in terms) * float(np.vdot(wide, wide).real)
        assert abs(s.expectation(terms) - want) <= 1e-13 * scale
        assert abs(s.expectation(terms[:n]) - sum(c * pauli_value(wide, t) for t, c in terms[:n])) <= 1e-13 * scale
        spins = np.array([[0.5 * pauli_value(wide, one(c, q)).real for c in "XYZ"] for q in range(n)])
        assert np.abs(s.spins() - spins).max() <= 1e-13


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,count", [(11, 64), (12, 1), (12, 63), (12, 64), (12, 65), (13, 64)])
def test_diagonal_strings_around_the_small_launch(pkg, precision, n, count):
    """The sizes and numbers of strings where one launch for a small state ends."""
    rng = np.random.default_rng(7 * n + count)
    a = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    a = (a / np.linalg.norm(a)).astype(np.complex128 if precision == 0 else np.complex64)
    wide = a.astype(np.complex128)
    strings = {"".join(rng.choice(list("IZ"), n)) for _ in range(2 * count)}
    terms = [(t, float(w)) for t, w in zip(sorted(strings)[:count], rng.standard_normal(count))]
    with pkg.State(n, precision) as s:
        s.upload(a)
        want = sum(c * pauli_value(wide, t) for t, c in terms)
        assert abs(s.expectation(terms) - want) <= 1e-13 * sum(abs(c) for _, c in terms) * float(np.vdot(wide, wide).real)
