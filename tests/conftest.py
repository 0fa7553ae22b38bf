import json
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "oracle"))

from __graft_entry__ import REFERENCE, load_package  # noqa: E402,F401  (REFERENCE: reference tree root)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200); runs through the C ABI of librbk.so")


# Modules and tests that fail without the reference's own build.
NEED_REFERENCE = {"test_gpu_bra_b200", "test_inner_product_pauli_vs_reference", "test_pauliss_hamiltonian_energy_full_precision"}


def pytest_collection_modifyitems(items):
    """Where the reference is not built, the tests that need it run after all others,
    so that a run that stops at its first failure has run those."""
    if not os.path.exists(os.path.join(ROOT, "oracle", "_ref", "libketref.so")):
        items.sort(key=lambda i: i.module.__name__ in NEED_REFERENCE or getattr(i, "originalname", "") in NEED_REFERENCE)


@pytest.fixture(scope="session")
def pkg():
    return load_package()


@pytest.fixture(scope="session")
def golden():
    d = os.path.join(ROOT, "tests", "golden")
    with open(os.path.join(d, "cases.json")) as f:
        meta = json.load(f)
    arrays = dict(np.load(os.path.join(d, "golden.npz")))
    return meta, arrays


def as_ops(ops_json):
    """cases.json stores instruction tuples as lists."""
    return [(m, tuple(q), tuple(p)) for m, q, p in ops_json]
