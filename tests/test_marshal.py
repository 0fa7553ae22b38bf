"""The native conversion of gate lists against the ctypes one: the same records,
and the same errors for malformed input (State.apply: test_marshal_apply.py)."""
import ctypes

import numpy as np
import pytest


@pytest.fixture
def plain(pkg, monkeypatch):
    """Runs a function with the ctypes conversion."""
    def run(fn, *args):
        with monkeypatch.context() as m:
            m.setattr(pkg.rbk, "marshal", lambda: None)
            return fn(*args)
    return run


def outcome(fn, *args):
    try:
        arr, count = fn(*args)[:2]
        return bytes(memoryview(arr).cast("B")) if count else b"", count
    except Exception as e:
        return type(e)


GOOD = [
    ("EX", (3,), 2, -0.5, ()),
    ("U3", [1], None, 0.0, (0.1, -2, np.float64(3.5))),
    ("CNOT", (np.int64(0), 4), None, 0, ()),
    ("U", (1, 2), None, 0.0, (-3,)),
    ("H", (7,), np.int32(5), 1, [1.0]),
    ("EZ", ("2", 1.0), "3", "0.25", ("1e-3",)),
]
BAD = [
    [("NOPE", (0,), None, 0.0, ())],
    [("H", ("x",), None, 0.0, ())],
    [("H", (0,), None, "x", ())],
    [("H", (0,), None, 0.0)],
    [("H", 0, None, 0.0, ())],
    [("EZ", (0,), "k", 1.0, ())],
]


@pytest.mark.parametrize("spec", [[], GOOD] + BAD)
def test_gate_lists(pkg, plain, spec):
    if not pkg.rbk.marshal():
        pytest.skip("the native conversion is not built")
    assert outcome(pkg.adjoint.gate_array, spec) == outcome(plain, pkg.adjoint.gate_array, spec)


class Growing(list):
    """A list that gets another gate when its first gate's qubit is read."""

    def __init__(self):
        outer = self

        class Qubit(int):
            def __int__(self):
                outer.append(("X", (1,), None, 0.0, ()))
                return 0
        super().__init__([("H", (Qubit(),), None, 0.0, ()), ("Y", (1,), None, 0.0, ())])


# Made anew for each conversion.
ODD = [
    lambda: [("H", (2 ** 31 + 1,), 2 ** 70, 1, ())], lambda: [("CNOT", np.array([3, 4, 5]), None, np.float32(0.5), np.arange(4.0))],
    lambda: [("H", {0}, None, 0.0, ())], lambda: [("H", {0: 1}, None, 0.0, ())], lambda: [("H", range(3), None, 0.0, [1, 2, 3, 4])],
    lambda: [("H", "12", None, "nan", "123")], lambda: [("H", (0,), None, 0.0, (), 1)], lambda: [iter(("H", (5,), None, 0.0, ()))],
    lambda: [(["H"], (0,), None, 0.0, ())], lambda: [("H", (0,), None, 10 ** 400, ())], lambda: [("EX", None, 0, 1.0, ())],
    lambda: [("EX", (0,), 0, 1.0, None)], lambda: {("H", (0,), None, 0.0, ()): 1}, lambda: (g for g in GOOD), lambda: None, Growing,
]


@pytest.mark.parametrize("k", range(len(ODD)))
def test_odd_gate_lists(pkg, plain, k):
    if not pkg.rbk.marshal():
        pytest.skip("the native conversion is not built")
    assert outcome(pkg.adjoint.gate_array, ODD[k]()) == outcome(plain, pkg.adjoint.gate_array, ODD[k]())
