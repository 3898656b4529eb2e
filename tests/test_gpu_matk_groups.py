"""Dense unitaries of 5 and more qubits on both sides of the line between a CTA a group and
tiles of groups: one group, the last number of groups that goes by itself, and the
first that does not, on scattered targets, against numpy."""
import numpy as np
import pytest

import ket_b200 as K
from ket_b200.circuit import DeviceState, KET_C64, KET_C128

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,groups", [(5, 0), (5, 11), (5, 12), (6, 9), (6, 10), (7, 0), (7, 9), (7, 10), (8, 8), (8, 9),
                                      (9, 7), (9, 8), (10, 0), (10, 7), (10, 8)])
@pytest.mark.parametrize("precision", [KET_C128, KET_C64])
def test_group_and_tile_kernels(k, groups, precision):
    n = k + groups
    r = np.random.default_rng(100 * k + groups)
    u = np.linalg.qr(r.normal(size=(1 << k, 1 << k)) + 1j * r.normal(size=(1 << k, 1 << k)))[0]
    q = [int(x) for x in r.permutation(n)[:k]]
    a = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    a /= np.linalg.norm(a)
    if precision == KET_C64:
        a = a.astype(np.complex64).astype(np.complex128)
    st = DeviceState(n, precision)
    st.set_amplitudes(a)
    st.apply_abi(*K.Circuit(n).unitary(u.tolist(), *q).to_abi(), prune=False)
    # axis n - 1 - q of the tensor is qubit q; q[0] is the matrix's most significant bit
    ax = [n - 1 - x for x in q]
    t = np.tensordot(u.reshape((2,) * (2 * k)), a.reshape((2,) * n), axes=(list(range(k, 2 * k)), ax))
    want = np.moveaxis(t, list(range(k)), ax).reshape(-1)
    # 2^k FP64 products a row of a unit vector, then the state's own rounding
    bound = 1e-14 if precision == KET_C128 else 2.0 ** -23
    assert np.abs(st.amplitudes_dense() - want).max() <= bound
