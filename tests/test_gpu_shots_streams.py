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
