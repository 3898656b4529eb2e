"""Dense unitaries on three to ten qubits: the register kernel (3 and 4 qubits)
and the shared-memory kernel (5 to 10), at the fewest groups, at a ragged number
of groups for a CTA, and with targets in any order, low and high."""
import numpy as np
import pytest

import ket_b200 as K
from ket_b200.circuit import DeviceState, KET_C64, KET_C128

pytestmark = pytest.mark.gpu


def dense_unitary(a, m, qs):
    n, k = a.size.bit_length() - 1, len(qs)
    axes = [n - 1 - q for q in qs]
    v = np.moveaxis(a.reshape([2] * n), axes, range(k))
    y = (m @ v.reshape(1 << k, -1)).reshape([2] * n)
    return np.moveaxis(y, range(k), axes).reshape(-1)


@pytest.mark.parametrize("precision", [KET_C128, KET_C64])
@pytest.mark.parametrize("k,extra", [(3, 0), (3, 1), (3, 9), (4, 0), (4, 8), (5, 0), (5, 3), (5, 9), (6, 1), (6, 7), (7, 2),
                                     (8, 1), (8, 5), (9, 4), (10, 0), (10, 3)])
def test_dense_unitary(k, extra, precision):
    n = k + extra
    r = np.random.default_rng(100 * k + extra)
    m = np.linalg.qr(r.normal(size=(1 << k, 1 << k)) + 1j * r.normal(size=(1 << k, 1 << k)))[0]
    a = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    a /= np.linalg.norm(a)
    if precision == KET_C64:
        a = a.astype(np.complex64).astype(np.complex128)
    for qs in (list(range(k)), list(range(n - 1, n - 1 - k, -1)), [int(q) for q in r.permutation(n)[:k]]):
        st = DeviceState(n, precision)
        st.set_amplitudes(a)
        st.apply_abi(*K.Circuit(n).unitary(m.tolist(), *qs).to_abi())
        # a row of 2^k products in FP64, then one rounding to the state's precision
        bound = 4 * 2.0 ** k * 2.0 ** -53 + (2.0 ** -23 if precision == KET_C64 else 0.0)
        assert np.abs(st.amplitudes_dense() - dense_unitary(a, m, qs)).max() <= bound
