"""Passes whose compiled kernels would outgrow the instruction cache are cut into
several: the state is the interpreter's, which takes them whole, bit for bit (the
cut stores and reloads the amplitudes unchanged; the circuits hold no controlled
phases, which merge by pass).  Deep circuits on the 12 qubits of one tile, at the
smallest size that is cut and on both sides of it, one of 1000 gates to cut in
many places, and a single gate that leaves nothing to cut."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _circuit(n, gates, seed):
    import ket_b200 as K
    r, c = random.Random(seed), K.Circuit(n)
    for _ in range(gates):
        a, b = r.sample(range(min(n, 12)), 2)
        k = r.randrange(9)
        if k < 3:
            c = c.rx(r.uniform(0, 6.28), a).rz(r.uniform(0, 6.28), a)
        elif k < 5:
            c = c.h(a).t(b)
        elif k == 5:
            c = c.ry(r.uniform(0, 6.28), a)
        elif k == 6:
            c = c.cnot(a, b)
        elif k == 7:
            c = c.swap(a, b)
        else:
            c = c.xx(r.uniform(0, 6.28), a, b)
    return c


@pytest.mark.parametrize("n,gates,precision,prune", [
    (21, 250, 0, True), (22, 1, 0, True), (22, 60, 0, False), (22, 250, 0, True), (22, 300, 1, True), (23, 1000, 0, False),
])
def test_cut_passes_equal_the_interpreter(n, gates, precision, prune):
    from ket_b200.circuit import DeviceState, flatten_ops, ops_to_abi
    arr, m, k = ops_to_abi(flatten_ops(_circuit(n, gates, n + gates).ops))
    out = []
    for specialize in (1, -1):
        st = DeviceState(n, precision=precision)
        st.set_basis(3)
        st.apply_abi(arr, m, k, prune=prune, specialize=specialize)
        out.append(st.amplitudes_dense())
    assert np.array_equal(out[0], out[1])


def test_kernels_compiled_ahead_match_the_cut_passes():
    """compile_kernels and the default policy cut alike: the circuit compiles nothing
    more when it runs, and its kernels are the ones that run."""
    import ctypes as C
    from ket_b200 import _lib
    from ket_b200.circuit import DeviceState, KET_C128

    def stats():
        s, t = (C.c_int64 * 4)(), C.c_double()
        _lib.check(_lib.lib().ket_jit_stats(s, C.byref(t)))
        return list(s)

    c = _circuit(22, 250, 5)
    assert c.compile_kernels(KET_C128, True) > 1
    before = stats()
    st = DeviceState(22, KET_C128)
    st.set_basis(0)
    st.apply_abi(*c.to_abi(), prune=True)
    got = st.amplitudes_dense()
    after = stats()
    assert after[0] == before[0] and after[3] > before[3]
    st.set_basis(0)
    st.apply_abi(*c.to_abi(), prune=True, specialize=-1)
    assert np.array_equal(got, st.amplitudes_dense())
