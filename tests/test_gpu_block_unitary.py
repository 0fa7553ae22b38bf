"""Dense block unitaries on CUDA cores (k = 1..6): states smaller than the
2^11-amplitude tile, of one tile and of several per CTA, targets on low, high and
mixed bits, after a SWAP that moves the layout map, against numpy in FP64.  The
products and sums are FP64: 64 terms of rounding 1e-16 (complex<double>), one
rounding of 6e-8 of an amplitude below 1 (complex<float>)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def apply_numpy(a, u, qubits, n):
    k = len(qubits)
    t = a.reshape([2] * n)
    axes = [n - 1 - q for q in reversed(qubits)]
    t = np.moveaxis(t, axes, list(range(k)))
    shp = t.shape
    t = (u @ t.reshape(1 << k, -1)).reshape(shp)
    return np.moveaxis(t, list(range(k)), axes).reshape(-1)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 3, 6, 8, 10, 11, 12, 20])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 6])
def test_block_unitary_vs_numpy(pkg, precision, n, k):
    if k > n or (precision == 1 and k >= 5 and n >= k + 7):  # the latter run on the tensor cores
        pytest.skip("not this path")
    rng = np.random.default_rng(100 * n + k)
    a = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    a = (a / np.linalg.norm(a)).astype(np.complex128 if precision == 0 else np.complex64)
    want = a.astype(np.complex128)
    with pkg.State(n, precision) as s:
        s.upload(a)
        for targets in (list(range(k)), list(range(n - k, n)), [int(x) for x in rng.permutation(n)[:k]]):
            z = rng.standard_normal((1 << k, 1 << k)) + 1j * rng.standard_normal((1 << k, 1 << k))
            u, _ = np.linalg.qr(z)
            s.apply_unitary(u, targets)
            want = apply_numpy(want, u, targets, n)
            if n > 1:
                s.swap(0, n - 1)
                want = np.swapaxes(want.reshape([2] * n), 0, n - 1).reshape(-1)
        got = s.amplitudes().astype(np.complex128)
    assert np.abs(got - want).max() <= (1e-14 if precision == 0 else 3e-7)
