"""Batched trajectories' start states in the xorshift32 stream: any number of draws a
shot (stepped one by one up to 64, by squaring from there on) and of shots, against
the generator itself."""
import numpy as np
import pytest

import ket_b200 as K
from ket_b200.circuit import make_prng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("measures", [1, 2, 31, 32, 62, 63, 64, 65, 100, 257])
@pytest.mark.parametrize("shots", [1, 3, 300])
def test_stream(measures, shots):
    """A qubit in |+>, measured again and again between H gates: outcome k of a shot is 1
    where its draw lies below P(1), which is 1/2 to rounding."""
    c = K.Circuit(1).creg("c", measures)
    for k in range(measures):
        c = c.h(0) if k == 0 else c.reset(0).h(0)
        c = c.measure(0, "c", k)
    idx, bits, layout, state = c.run_shots(shots=shots, seed=1234)
    rng = make_prng(1234)
    want = np.zeros((shots, measures), dtype=np.uint8)
    for s in range(shots):
        one = None
        for k in range(measures):
            if k:
                rng()  # the reset's draw
            want[s, k] = rng() < 0.5
        rng()  # the sample's
    assert np.array_equal(bits, want)
    assert np.array_equal(np.asarray(idx), want[:, -1]) and state == rng.state[0]


@pytest.mark.parametrize("n,rounds,noise", [(3, 120, (0.0, 0.0, 0.0)), (4, 90, (0.1, 0.2, 0.1)), (7, 150, (0.02, 0.05, 0.0)),
                                            (10, 160, (0.01, 0.02, 0.1)), (12, 80, (0.0, 0.0, 0.1))])
def test_many_segments(n, rounds, noise):
    """A measurement or reset after every few gates, more segments than shared memory holds at
    a time, and runs of gates between them whose noise makes the next draw a jump, against
    the oracle shot by shot."""
    from oracle import oracle as O
    from test_gpu_shots_rounds import raw
    r = np.random.default_rng(n)
    c, o = K.Circuit(n).creg("c", 3), O.OCircuit(n)
    for k in range(rounds):
        for _ in range(40 if k % 29 == 28 else int(r.integers(1, 4))):
            a, b = (int(q) for q in r.permutation(n)[:2])
            g = int(r.integers(0, 4))
            t = float(r.uniform(0, 6.28))
            if g == 0:
                c = c.ry(t, a)
                o.add("ry", [a], [t])
            elif g == 1:
                c = c.cnot(a, b)
                o.add("cnot", [a, b])
            elif g == 2:
                c = c.h(a)
                o.add("h", [a])
            else:
                c = c.xx(t, a, b)
                o.add("xx", [a, b], [t])
        a, bit = int(r.integers(n)), int(r.integers(3))
        if k % 4 == 3:
            c = c.reset(a)
            o.reset(a)
        else:
            c = c.measure(a, "c", bit)
            o.measure(a, bit)
    shots = 20
    idx, bits, state = raw(c, 0, 2, shots, noise)
    oidx, obits, ostate = o.run_pershot(shots, 77, *noise, ncbits=3)
    assert np.array_equal(idx, oidx) and np.array_equal(bits.reshape(shots, 3), obits) and state == ostate
