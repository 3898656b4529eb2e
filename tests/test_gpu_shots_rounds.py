"""Batched trajectories (rounds, relabellings, Pauli frames) against one
trajectory at a time through the fused engine, shot by shot: one to thirteen
qubits, both precisions, strong noise between gates of every kind, gates and swaps
in if-bodies, and programs longer than a segment."""
import ctypes as C

import numpy as np
import pytest

import ket_b200 as K

pytestmark = pytest.mark.gpu


def circuit(n, depth, seed):
    r = np.random.default_rng(seed)
    u = {k: np.linalg.qr(r.normal(size=(1 << k, 1 << k)) + 1j * r.normal(size=(1 << k, 1 << k)))[0].tolist() for k in (1, 2, 3, 4)}
    c = K.Circuit(n)
    for i in range(depth):
        k = str(r.choice(["h", "t", "y", "rx", "ry", "rz", "u3", "cnot", "cnot", "cnot", "swap", "cz", "crx", "cu3", "xx", "xy",
                          "ccx", "cswap", "csrswap", "u", "measure", "reset", "if"]))
        q = [int(x) for x in r.permutation(n)]
        a = r.uniform(0, 6.28, 3).tolist()
        need = {"ccx": 3, "cswap": 3, "csrswap": 3}.get(k, 2 if k in ("cnot", "swap", "cz", "crx", "cu3", "xx", "xy") else 1)
        if need > n:
            continue
        if k == "u":
            w = int(r.integers(1, min(4, n) + 1))
            c = c.unitary(u[w], *q[:w])
        elif k == "measure":
            c = c.measure(q[0], "c", int(r.integers(3)))
        elif k == "reset":
            c = c.reset(q[0])
        elif k == "if":  # (no draw in it: the noise acts on gates of one and two qubits)
            if n >= 3:
                c = c.if_("c", int(r.integers(4)), lambda b: b.ccx(*q[:3]).cswap(*q[:3]) if seed % 2 else b.ccx(*q[:3]))
        elif k in ("rx", "ry", "rz", "crx", "xx", "xy"):
            c = getattr(c, k)(a[0], *q[:need])
        elif k in ("u3", "cu3"):
            c = getattr(c, k)(*a, *q[:need])
        else:
            c = getattr(c, k)(*q[:need])
    return c


def raw(c, precision, path, shots, noise):
    from ket_b200 import _lib
    from ket_b200.circuit import DeviceState, shots_to_abi
    arr, m, k, nb, _ = shots_to_abi(c.ops, c._cregs)
    st = DeviceState(c.qubits, precision)
    state = C.c_uint32(77)
    idx, bits = np.zeros(shots, dtype=np.uint64), np.zeros(max(shots * nb, 1), dtype=np.uint8)
    mv = np.ascontiguousarray(m).view(np.float64)
    _lib.check(_lib.lib().ket_debug_pershot_path(path))
    try:
        _lib.check(_lib.lib().ket_run_shots(st.h, arr, k, mv.ctypes.data_as(C.POINTER(C.c_double)), m.size,
                                            C.byref(_lib.ket_noise(*noise)), 0, shots, C.byref(state), nb,
                                            idx.ctypes.data_as(C.POINTER(C.c_uint64)),
                                            bits.ctypes.data_as(C.POINTER(C.c_uint8))))
    finally:
        _lib.lib().ket_debug_pershot_path(0)
    return idx, bits, state.value


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,depth,noise", [(1, 30, (0.2, 0.0, 0.1)), (2, 40, (0.2, 0.2, 0.0)), (3, 60, (0.1, 0.3, 0.1)),
                                           (4, 80, (0.0, 0.0, 0.0)), (5, 80, (0.1, 0.2, 0.0)), (6, 500, (0.02, 0.05, 0.1)),
                                           (9, 120, (0.05, 0.1, 0.0)), (10, 150, (0.05, 0.1, 0.1)), (11, 90, (0.0, 0.2, 0.0)),
                                           (12, 700, (0.01, 0.02, 0.05)), (13, 120, (0.05, 0.1, 0.0))])
def test_batched_matches_one_at_a_time(n, depth, noise, precision):
    if n == 13 and precision == 0:
        pytest.skip("thirteen qubits are batched at c64 only")
    for seed in (1, 2):
        c = circuit(n, depth, 100 * n + seed)
        a, b = raw(c, precision, 2, 24, noise), raw(c, precision, 1, 24, noise)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2] == b[2]
