"""The default options find the kernels that were compiled before, below 26 qubits too,
and those compiled for other programs change nothing."""
import ctypes as C

import numpy as np
import pytest

import ket_b200 as K
from ket_b200 import _lib
from ket_b200 import workloads as W
from ket_b200.circuit import DeviceState, flatten_ops, ops_to_abi

pytestmark = pytest.mark.gpu


def launches():
    return _lib.jit_stats()["launches"]


def run(n, abi, precision=0, **kw):
    st = DeviceState(n, precision)
    st.set_basis(0)
    at = launches()
    st.apply_abi(*abi, **kw)
    return st.amplitudes_dense(), launches() - at


def compile_only(n, abi, precision=0, **kw):
    arr, m, k = abi
    mv = np.ascontiguousarray(m).view(np.float64)
    o = _lib.exec_opts(**kw)
    kernels = C.c_int64()
    _lib.check(_lib.lib().ket_jit_compile(n, precision, arr, k, mv.ctypes.data_as(C.POINTER(C.c_double)), m.size,
                                          C.byref(o), C.byref(kernels), None, 0))
    return kernels.value


def long_circuit(n, layers, seed):
    """Layers on ten of the qubits: a pass of hundreds of gates, without phases to merge."""
    r = np.random.default_rng(seed)
    c = K.Circuit(n)
    for _ in range(layers):
        for q in range(10):
            c = c.ry(float(r.uniform(0, 6)), q).rx(float(r.uniform(0, 6)), q)
        for q in range(9):
            c = c.cnot(q, q + 1)
    return c


@pytest.mark.parametrize("n", [22, 25])
@pytest.mark.parametrize("precision", [0, 1])
def test_kernels_of_cut_passes_serve_the_default_policy(n, precision):
    """specialize = 1 cuts its long passes; the call after it with the default options
    has to cut them alike."""
    abi = long_circuit(n, 8, n + precision).to_abi()
    want, ran = run(n, abi, precision, specialize=1)
    assert ran > 1
    got, again = run(n, abi, precision)
    assert again == ran and np.array_equal(got, want)


@pytest.mark.parametrize("n", [13, 16])
def test_kernels_for_other_register_bits_are_not_waited_for(n):
    """Kernels compiled for 4 register bits serve no default call below 26 qubits: such a
    call still runs in one launch."""
    c, _ = W.brickwork_circuit(n, 6, 40 + n)
    abi = c.to_abi()
    want, _ = run(n, abi)
    assert compile_only(n, abi, reg_bits=4) >= 1
    got, ran = run(n, abi)
    assert ran == 0 and np.array_equal(got, want)


def test_kernels_for_other_matrices_are_not_waited_for():
    """The same gates with matrices of another form (real in place of general) need other
    kernels."""
    n = 14
    def circuit(general):
        c = K.Circuit(n)
        for layer in range(4):
            for q in range(n):
                c = c.u3(0.3 + q, 0.7 if general else 0.0, 0.2 if general else 0.0, q)
            for q in range(n - 1):
                c = c.cnot(q, q + 1)
        return c.to_abi()
    want, _ = run(n, circuit(False))
    assert compile_only(n, circuit(True)) >= 1
    got, ran = run(n, circuit(False))
    assert ran == 0 and np.array_equal(got, want)
    _, ran = run(n, circuit(True))
    assert ran > 0


def test_compiled_ahead_with_default_options_still_serves():
    c, _ = W.brickwork_qft(14, 5, 91)
    abi = ops_to_abi(flatten_ops(c.ops))
    assert compile_only(14, abi) >= 1
    got, ran = run(14, abi)
    want, _ = run(14, abi, specialize=-1)
    assert ran > 0 and np.array_equal(got, want)


def test_whole_passes_until_kernels_are_ready():
    """From 26 qubits on a default call whose cut passes still wait for their kernels takes
    the whole passes on the interpreter; once the kernels are ready it runs those."""
    n = 26
    abi = long_circuit(n, 10, 77).to_abi()
    want, ran = run(n, abi, specialize=-1)
    assert ran == 0
    first, ran = run(n, abi)
    assert ran == 0 and np.array_equal(first, want)
    _lib.check(_lib.lib().ket_jit_wait())
    got, ran = run(n, abi)
    assert ran > 1 and np.array_equal(got, want)


@pytest.mark.parametrize("precision,prune,cut", [(0, True, False), (0, False, True), (1, True, True)])
def test_passes_beyond_a_kernel(precision, prune, cut):
    """More ops than a compiled kernel holds: cut for kernels, or one pass of the interpreter
    where that is the faster (complex128 with pruning)."""
    n = 22
    abi = long_circuit(n, 27, 5).to_abi()
    want, _ = run(n, abi, precision, prune=prune, specialize=-1)
    got, ran = run(n, abi, precision, prune=prune, specialize=1)
    assert (ran > 1 if cut else ran == 0) and np.array_equal(got, want)
