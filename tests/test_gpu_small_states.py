"""complex128 circuits on up to 20 qubits in one launch (the automatic path there) against one
gate a launch: below, at and above one tile, every kind of gate between
relabellings, with and without pruning, from any basis state;
and against the register-tiled passes on the reference's benchmark families."""
import numpy as np
import pytest

import ket_b200 as K
from ket_b200 import workloads as W
from ket_b200.algorithms import qft
from ket_b200.circuit import DeviceState, KET_C64, KET_C128

pytestmark = pytest.mark.gpu


def circuit(n, depth, seed):
    r = np.random.default_rng(seed)
    u = {k: np.linalg.qr(r.normal(size=(1 << k, 1 << k)) + 1j * r.normal(size=(1 << k, 1 << k)))[0].tolist() for k in (1, 2, 3, 4, 5)}
    c = K.Circuit(n)
    for _ in range(depth):
        k = str(r.choice(["h", "t", "x", "y", "z", "rx", "ry", "rz", "u3", "cnot", "cnot", "cnot", "swap", "cz", "cu1", "crx",
                          "crz", "cu3", "xx", "zz", "xy", "ccx", "cswap", "csrswap", "u"]))
        q = [int(x) for x in r.permutation(n)]
        a = r.uniform(0, 6.28, 3).tolist()
        need = 3 if k in ("ccx", "cswap", "csrswap") else 2 if k in ("cnot", "swap", "cz", "cu1", "crx", "crz", "cu3", "xx", "zz", "xy") else 1
        if need > n:
            continue
        if k == "u":
            w = int(r.integers(1, min(4, n) + 1))
            c = c.unitary(u[w], *q[:w])
        elif k in ("rx", "ry", "rz", "cu1", "crx", "crz", "xx", "zz", "xy"):
            c = getattr(c, k)(a[0], *q[:need])
        elif k in ("u3", "cu3"):
            c = getattr(c, k)(*a, *q[:need])
        else:
            c = getattr(c, k)(*q[:need])
    return c, u


def run(c, precision, prune, fusion, init, specialize=0):
    st = DeviceState(c.qubits, precision)
    st.set_basis(init)
    st.apply_abi(*c.to_abi(), fusion=fusion, prune=prune, specialize=specialize)
    return st.amplitudes_dense()


@pytest.mark.parametrize("n,depth", [(1, 12), (2, 30), (3, 60), (4, 80), (5, 300), (8, 200), (11, 150), (12, 150), (13, 150), (14, 90),
                                     (17, 120), (19, 100), (20, 120)])
def test_one_launch_matches_gate_by_gate(n, depth):
    for prune in (True, False):
        c, _ = circuit(n, depth, 1000 * n + prune)
        init = (1 << n) - 1 if prune else 0
        a, b = run(c, KET_C128, prune, -1, init), run(c, KET_C128, prune, 0, init)
        # rounding of `depth` gates of a unit vector, and of folded factors
        assert np.abs(a - b).max() <= depth * 1e-15


@pytest.mark.parametrize("n", [3, 12, 16])
def test_complex64_keeps_the_passes(n):
    """complex64 results are those of the interpreter's passes, bit for bit."""
    c, _ = circuit(n, 60, n)
    assert np.array_equal(run(c, KET_C64, True, -1, 0), run(c, KET_C64, True, -1, 0, specialize=-1))


def test_relabellings_alone_and_wide_unitaries():
    for n in (3, 12, 15):
        c = K.Circuit(n).x(0).cnot(0, n - 1).swap(1, n - 1).x(n - 1).cnot(n - 1, 0)
        assert np.array_equal(run(c, KET_C128, True, -1, 5), run(c, KET_C128, True, 0, 5))
    c, u = circuit(14, 30, 4)
    c = c.unitary(u[5], 3, 9, 0, 13, 6).h(2)  # wider than the one launch takes: the passes run it
    assert np.abs(run(c, KET_C128, True, -1, 0) - run(c, KET_C128, True, 0, 0)).max() <= 1e-13


@pytest.mark.parametrize("n", [10, 16, 20])
def test_one_launch_matches_tiled_passes(n):
    c = W.brickwork_circuit(n, 12, 7)[0].append(qft(n))
    for prune in (True, False):
        a, b = run(c, KET_C128, prune, -1, 0), run(c, KET_C128, prune, -1, 0, specialize=-1)
        assert np.abs(a - b).max() <= 1e-13
