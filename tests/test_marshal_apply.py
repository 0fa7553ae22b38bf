"""State.apply through the native conversion against the ctypes calls, both into
recorders in place of the library's entry points: the same calls in the same
order, and the same exception at the same instruction."""
import ctypes

import numpy as np
import pytest


class Recorder:
    """ctypes functions with the entry points' signatures that note their arguments."""

    def __init__(self, rbk, fail_after=None):
        self.calls, self.functions = [], {}
        for name in rbk._MARSHALLED:
            argtypes, restype = rbk._SIGNATURES[name]
            self.functions[name] = ctypes.CFUNCTYPE(restype, *argtypes)(self.note(name, argtypes, fail_after))

    def note(self, name, argtypes, fail_after):
        def call(*args):
            values = []
            for k, (a, t) in enumerate(zip(args, argtypes)):
                if t is ctypes.POINTER(ctypes.c_uint32):
                    values.append([a[i] for i in range(args[k + 1])])
                else:
                    values.append(a)
            self.calls.append((name, values))
            return 1 if fail_after is not None and len(self.calls) > fail_after else 0
        return call

    def __getattr__(self, name):
        if name == "rbk_last_error":
            return lambda: b"recorded"
        return self.functions[name]


@pytest.fixture
def both(pkg, monkeypatch):
    """Runs ops (made anew by `make(state)` each time) natively and through ctypes; the two outcomes."""
    rbk = pkg.rbk
    if not rbk.marshal():
        pytest.skip("the native conversion is not built")

    def bind(table):
        rbk._native.bind([ctypes.cast(getattr(table, n), ctypes.c_void_p).value for n in rbk._MARSHALLED])

    def run(make, handle=0x1000, fail_after=None):
        outcomes = []
        for native in (True, False):
            rec = Recorder(rbk, fail_after)
            s = object.__new__(rbk.State)
            s.h = ctypes.c_void_p(handle) if handle else None
            error = None
            with monkeypatch.context() as m:
                m.setattr(rbk, "lib", lambda: rec)
                if native:
                    bind(rec)
                else:
                    m.setattr(rbk, "marshal", lambda: False)
                try:
                    s.apply(make(s))
                except Exception as e:
                    error = type(e)
                finally:
                    s.h = None  # nothing to destroy
                    if native:
                        bind(pkg.rbk._lib)
            outcomes.append((rec.calls, error))
        return outcomes

    pkg.rbk.lib()
    yield run


ITERATOR = ("H", (0,), ())  # handed over as an iterator
EVERY = [
    ("H", (0,), ()), ("X", (1,), ()), ("Y", (2,), ()), ("Z", (3,), ()), ("U1", (4,), (0.5,)), ("U2", (5,), (0.1, -0.2)),
    ("U3", (6,), (0.1, 0.2, 0.3)), ("CNOT", (0, 1), ()), ("CZ", (2, 3), ()), ("U", (4, 5), (-3,)), ("EX", (0,), (1.0,)),
    ("EY", (1,), (2,)), ("EZ", (2,), (3.5,)), ("SWAP", (0, 1), ()), ("BEGIN FUSION", (), ()), ("END FUSION", (), ()),
]
ODD = [
    ("H", (0,), None), ("X", [1, 9], 7), ("BEGIN FUSION", None, None), ["CNOT", [0, 1], None],  # operands that are not used
    ("H", np.array([3]), ()), ("CZ", np.array([3, 4]), np.zeros(0)), ("CNOT", {0: 5, 1: 6}, ()), ("H", range(4, 6), ()),
    ("H", (np.int64(2),), ()), ("H", (True,), ()), ("H", (-1,), ()), ("H", (2 ** 32 + 1,), ()), ("H", (2 ** 70,), ()),
    ("Z", (1.0,), ()), ("CZ", ("3", 2.0), ()), ("U1", (1.5,), (0.5,)), ("CNOT", (1.0, 2), ()),  # int(q) takes these
    ("U3", (0,), np.array([1, 2, 3], np.float32)), ("EX", (0,), (np.float64(0.5),)), ("EX", (0,), (ctypes.c_double(0.5),)),
    ("H", (ctypes.c_uint32(3),), ()), ("U", (0, 1), ("4",)), ("U", (0, 1), (2.9,)), ("U", (0, 1), (2 ** 70 + 3,)),
    (np.str_("H"), (0,), ()), ITERATOR, ("EX", (0,), {0: 0.25}),
]
BAD = [
    ("H", (0.5,), ()), ("H", ("0",), ()), ("H", (None,), ()), ("H", (), ()), ("H", 0, ()), ("H", {0, 1}, ()), ("H", None, ()),
    ("CNOT", (0,), ()), ("CZ", (0,), ()), ("U1", (0,), ()), ("U1", (0,), ("0.5",)), ("U1", (0,), (1j,)), ("U1", (0,), None),
    ("U3", (0,), (1, 2)), ("U", (0, 1), ("x",)), ("U", (0, 1), (float("nan"),)), ("NOPE", (0,), ()), ("H\0", (0,), ()),
    (b"H", (0,), ()), (3, (0,), ()), ("H", (0,)), ("H", (0,), (), ()), 5, None, "abc", "ab", ("EX", (0,), (10 ** 400,)),
]


@pytest.mark.parametrize("k", range(len(EVERY + ODD + BAD)))
def test_one_instruction(both, k):
    op = (EVERY + ODD + BAD)[k]
    native, plain = both(lambda _: [("X", (7,), ()), op if op is not ITERATOR else iter(op), ("Y", (8,), ())])
    assert native == plain
    assert len(plain[0]) == (3 if k < len(EVERY + ODD) else 1)


@pytest.mark.parametrize("make", [
    lambda s: EVERY, lambda s: tuple(EVERY), lambda s: iter(EVERY), lambda s: {("H", (0,), ()): 1}, lambda s: [], lambda s: (),
    lambda s: None, lambda s: 5, lambda s: (op for op in EVERY + [("H", (), ())] + EVERY)])
def test_sequences(both, make):
    native, plain = both(make)
    assert native == plain


def test_generator_that_raises_midway(both):
    def make(_):
        yield ("H", (0,), ())
        yield ("X", (1,), ())
        raise OSError
    native, plain = both(make)
    assert native == plain and plain[1] is OSError and len(plain[0]) == 2


def test_state_closed_before_and_midway(both):
    native, plain = both(lambda s: EVERY, handle=None)
    assert native == plain

    def make(s):
        yield ("H", (0,), ())
        s.h = None
        yield ("X", (1,), ())
    native, plain = both(make)
    assert native == plain and plain[0][1][1][0] is None


def test_failing_call_ends_the_sequence(both, pkg):
    native, plain = both(lambda s: EVERY, fail_after=4)
    assert native == plain and plain[1] is pkg.RbkError and len(plain[0]) == 5


def test_instructions_changed_while_they_are_applied(both):
    class Index:
        def __init__(self, ops):
            self.ops = ops

        def __index__(self):
            self.ops.append(("Y", (1,), ()))
            return 2

    def make(_):
        ops = [("H", (0,), ())]
        ops.append(("X", [Index(ops)], ()))
        return ops
    native, plain = both(make)
    assert native == plain and len(plain[0]) == 3
