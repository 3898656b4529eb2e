"""The one-launch path of complex128 circuits of up to 20 qubits where it cannot run as
usual: a device without room for all its CTAs leaves the circuit to the passes, and a
grid barrier that gives up is reported and leaves the context usable."""
import numpy as np
import pytest

import ket_b200 as K
from ket_b200 import _lib
from ket_b200 import workloads as W
from ket_b200.circuit import DeviceState

pytestmark = pytest.mark.gpu


def run(c, **kw):
    st = DeviceState(c.qubits)
    st.set_basis(0)
    st.apply_abi(*c.to_abi(), **kw)
    return st.amplitudes_dense()


@pytest.fixture
def hook():
    L = _lib.lib()
    yield lambda *a: _lib.check(L.ket_debug_rounds_hook(*a))
    _lib.check(L.ket_debug_rounds_hook(0, 0))


# CTAs of a launch: 1 up to 12 qubits, 8 at 13, 64 at 16, 256 at 20
@pytest.mark.parametrize("n,ctas", [(13, 8), (16, 64), (18, 128), (20, 256)])
def test_no_room_for_the_grid(hook, n, ctas):
    c, _ = W.brickwork_circuit(n, 6, 5)
    one, passes = run(c), run(c, specialize=-1)
    assert np.abs(one - passes).max() <= 1e-13
    hook(ctas, 0)
    assert np.array_equal(run(c), one)
    hook(ctas - 1, 0)
    assert np.array_equal(run(c), passes)


def test_one_cta_needs_no_room(hook):
    c, _ = W.brickwork_circuit(12, 6, 5)
    one = run(c)
    hook(1, 0)
    assert np.array_equal(run(c), one)


def test_barrier_times_out_and_recovers(hook):
    c, _ = W.brickwork_circuit(20, 8, 5)
    want = run(c)
    hook(0, 1)
    with pytest.raises(K.KetError) as ei:
        run(c)
    assert ei.value.code == _lib.KET_ERR_TIMEOUT
    hook(0, 0)
    assert np.array_equal(run(c), want)
