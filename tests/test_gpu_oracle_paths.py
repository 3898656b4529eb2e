"""The paths that small complex128 circuits no longer take by default, and the batched
trajectories, against the CPU oracle.

Circuits of up to 20 qubits run in one launch unless told otherwise; the register-tiled
passes of larger states are checked here on the same sizes, interpreted, compiled and
compiled for 4 register bits, with every kind of gate.  The trajectories share their
planner with that launch, so they are checked shot by shot against the oracle's."""
import numpy as np
import pytest

from test_gpu_parity import AMP_TOL, build_both, random_gates
from test_gpu_shots_rounds import raw

pytestmark = pytest.mark.gpu

PASSES = [dict(specialize=-1), dict(specialize=1), dict(specialize=1, reg_bits=4)]


def amplitudes(kc, init, prune, **kw):
    from ket_b200.circuit import DeviceState, flatten_ops, ops_to_abi
    st = DeviceState(kc.qubits)
    st.set_basis(init)
    st.apply_abi(*ops_to_abi(flatten_ops(kc.ops)), prune=prune, **kw)
    return st.amplitudes_dense()


@pytest.mark.parametrize("n,seed", [(12, 31), (13, 32), (15, 33), (17, 34)])
@pytest.mark.parametrize("prune", [True, False])
def test_passes_of_random_gates(n, seed, prune):
    from oracle import oracle as O
    kc, oc = build_both(n, random_gates(n, 90 + 5 * n, seed, unitary=prune))
    init = seed * 331 % (1 << n) if prune else 0
    want = oc.simulate(init=init, mode=O.DENSE_PRUNE if prune else O.DENSE).dense()
    for kw in PASSES:
        assert np.max(np.abs(amplitudes(kc, init, prune, **kw) - want)) < AMP_TOL, kw


def test_passes_of_brickwork_qft():
    from ket_b200 import workloads as W
    from oracle import oracle as O
    kc, _ = W.brickwork_qft(20, 20, 17)
    oc, _ = O.brickwork(20, 20, 17, with_qft=True)
    want = oc.simulate(mode=O.DENSE_PRUNE).dense()
    for kw in PASSES:
        assert np.max(np.abs(amplitudes(kc, 0, True, **kw) - want)) < AMP_TOL, kw


def trajectory_circuits(n, depth, seed):
    """The same circuit for the engine and for the oracle: gates of every kind between
    measurements, resets and ifs without draws."""
    import ket_b200 as K
    from oracle import oracle as O
    r = np.random.default_rng(seed)
    c, o = K.Circuit(n).creg("c", 3), O.OCircuit(n)
    one, two, three = ["h", "t", "y", "x", "s", "v"], ["cnot", "cnot", "swap", "cz", "ch", "iswap"], ["ccx", "cswap", "csrswap"]
    angles = {"rx": (1, 1), "ry": (1, 1), "rz": (1, 1), "u3": (3, 1), "crx": (1, 2), "crz": (1, 2), "xx": (1, 2), "xy": (1, 2),
              "cu3": (3, 2)}
    for _ in range(depth):
        q = [int(x) for x in r.permutation(n)]
        k = str(r.choice(one + two + three + list(angles) + ["unitary", "measure", "reset", "if"]))
        need = 3 if k in three or k == "if" else 2 if k in two else angles[k][1] if k in angles else 1
        if need > n:
            continue
        if k == "unitary":
            w = int(r.integers(1, min(4, n) + 1))
            u = np.linalg.qr(r.normal(size=(1 << w, 1 << w)) + 1j * r.normal(size=(1 << w, 1 << w)))[0]
            c = c.unitary(u.tolist(), *q[:w])
            o.unitary(u.tolist(), q[:w])
        elif k == "measure":
            b = int(r.integers(3))
            c = c.measure(q[0], "c", b)
            o.measure(q[0], b)
        elif k == "reset":
            c = c.reset(q[0])
            o.reset(q[0])
        elif k == "if":
            v = int(r.integers(4))
            body = O.OCircuit(n)
            body.add("ccx", q[:3])
            body.add("cswap", q[:3])
            c = c.if_("c", v, lambda b: b.ccx(*q[:3]).cswap(*q[:3]))
            o.if_(0, 3, v, body)
        else:
            p = [float(x) for x in r.uniform(0, 6.28, angles[k][0])] if k in angles else []
            c = getattr(c, k)(*p, *q[:need])
            o.add(k, q[:need], p)
    return c, o


@pytest.mark.parametrize("n,depth,noise", [(1, 30, (0.2, 0.0, 0.1)), (2, 40, (0.2, 0.2, 0.0)), (3, 60, (0.1, 0.3, 0.1)),
                                           (4, 80, (0.0, 0.0, 0.0)), (5, 80, (0.1, 0.2, 0.0)), (7, 300, (0.02, 0.05, 0.1)),
                                           (10, 120, (0.05, 0.1, 0.1)), (12, 60, (0.05, 0.1, 0.05))])
def test_batched_trajectories(n, depth, noise):
    shots = 24
    for seed in (5, 6):
        c, o = trajectory_circuits(n, depth, 100 * n + seed)
        idx, bits, state = raw(c, 0, 2, shots, noise)
        oidx, obits, ostate = o.run_pershot(shots, 77, *noise, ncbits=3)
        assert np.array_equal(idx, oidx) and np.array_equal(bits.reshape(shots, 3), obits) and state == ostate
