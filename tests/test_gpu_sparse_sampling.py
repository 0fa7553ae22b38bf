"""Sampling at the edges of the two-level prefix sums (blocks of 128 amplitudes,
chunks of 4096): states smaller than a block, of one chunk and of several, with
most amplitudes zero, so that whole blocks and chunks have no weight.  The events
equal the oracle's, which walks the prefix sums of every amplitude; an event can
differ only where its draw lies within rounding of a bin edge (1e-13 an event)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 6, 7, 8, 11, 12, 13, 17])
def test_sparse_state_events_vs_oracle(pkg, n):
    rng = np.random.default_rng(n)
    a = np.zeros(1 << n, dtype=np.complex128)
    where = rng.permutation(1 << n)[:max(1, (1 << n) // 100)]
    a[where] = rng.standard_normal(where.size) + 1j * rng.standard_normal(where.size)
    a /= np.linalg.norm(a)
    with pkg.State(n) as s:
        s.upload(a)
        o = oracle.COracle(n)
        o.set_amplitudes(a)
        for num in (1, 5, 3000):
            ev = s.generate_events(num, 7 + num)
            assert np.array_equal(ev, o.generate_events(num, 7 + num))
            assert np.all(np.abs(a[ev]) > 0)


def test_sparse_chunks_vs_oracle(pkg):
    """24 qubits: four chunks per thread of the scan, 19 of 20 of weight zero."""
    n = 24
    rng = np.random.default_rng(n)
    a = np.zeros((1 << (n - 12), 4096), dtype=np.complex128)
    chunks = rng.permutation(a.shape[0])[:a.shape[0] // 20]
    a[chunks[:, None], rng.integers(4096, size=(chunks.size, 3))] = 10.0 ** rng.uniform(-6, 0, (chunks.size, 3))
    a = a.ravel() / np.linalg.norm(a)
    with pkg.State(n) as s:
        s.upload(a)
        o = oracle.COracle(n)
        o.set_amplitudes(a)
        ev = s.generate_events(5000, 3)
        assert np.array_equal(ev, o.generate_events(5000, 3))
        assert np.all(np.abs(a[ev]) > 0)
