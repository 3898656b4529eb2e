"""The one launch of small complex128 states stores its last pass in logical order: circuits
that only relabel, and gates between relabellings, on one tile and on grids of each
size, from random states."""
import numpy as np
import pytest

import ket_b200 as K
from ket_b200.circuit import DeviceState

pytestmark = pytest.mark.gpu


def run(c, a, **kw):
    st = DeviceState(c.qubits)
    st.set_amplitudes(a)
    st.apply_abi(*c.to_abi(), prune=False, **kw)
    return st.amplitudes_dense()


def state(n):
    r = np.random.default_rng(n)
    a = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    return a / np.linalg.norm(a)


def shuffle(c, r, count):
    n = c.qubits
    for _ in range(count):
        a, b = (int(q) for q in r.permutation(n)[:2])
        k = int(r.integers(0, 4))
        c = c.cnot(a, b) if k < 2 else c.swap(a, b) if k == 2 else c.x(a)
    return c


@pytest.mark.parametrize("n", [2, 4, 5, 8, 9, 10, 11, 12, 13, 14, 16, 17, 18, 19, 20])
def test_relabellings_alone(n):
    a, r = state(n), np.random.default_rng(100 + n)
    for c in (K.Circuit(n).x(n - 1), K.Circuit(n).cnot(0, n - 1), K.Circuit(n).swap(0, n - 1), shuffle(K.Circuit(n), r, 3 * n)):
        assert np.array_equal(run(c, a), run(c, a, fusion=0))


@pytest.mark.parametrize("n", [2, 4, 8, 9, 11, 12, 13, 15, 17, 18, 19, 20])
def test_gates_between_relabellings(n):
    a, r = state(n), np.random.default_rng(200 + n)
    c = K.Circuit(n)
    for _ in range(6):  # several passes from 13 qubits on
        for q in r.permutation(n):
            c = c.ry(float(r.uniform(0, 6)), int(q))
        c = shuffle(c, r, n)
    for tail in (c, c.h(0), c.rz(0.3, n - 1)):
        # rounding of at most 6 n gates of a unit vector, and of folded factors
        assert np.abs(run(tail, a) - run(tail, a, fusion=0)).max() <= 6 * n * 1e-15
