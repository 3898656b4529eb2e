"""Which Pauli terms go by tiles and which by their own pass: one flip mask in all, with as
many terms as a pass of its own takes as parameters, as a tile takes, and more, on both
sides of the width where the rule ends, and more flip masks than the planner looks
ahead over."""
import numpy as np
import pytest

from ket_b200.circuit import DeviceState
from test_gpu_pauli_tile import energy, word

pytestmark = pytest.mark.gpu


def state(n, r):
    a = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    a /= np.linalg.norm(a)
    st = DeviceState(n)
    st.set_amplitudes(a)
    return a, st


def check(a, st, terms):
    # FP64 products and sums of a unit vector: a few hundred roundings at most on any path to the result
    assert abs(st.expect_pauli_sum(terms) - energy(a, terms)) <= 1e-13 * sum(abs(c) for c, _ in terms)


@pytest.mark.parametrize("n", [12, 15])
@pytest.mark.parametrize("count", [1, 2, 64, 65, 512, 513])
@pytest.mark.parametrize("flips", [(), (0,), (2, 9), (11,)])
def test_one_flip_mask(n, count, flips):
    r = np.random.default_rng(1000 * n + count + len(flips))
    a, st = state(n, r)
    terms = []
    for _ in range(count):
        at = {q: "Z" for q in range(n) if q not in flips and r.random() < 0.5}
        for q in flips:
            at[q] = "X"
        terms.append((float(r.normal()), word(n, at or {0: "Z"})))
    check(a, st, terms)


@pytest.mark.parametrize("n", [20, 21])
def test_either_side_of_the_rule(n):
    r = np.random.default_rng(n)
    a, st = state(n, r)
    one = [(0.7, word(n, {3: "X", n - 1: "Y"}))]
    check(a, st, one)
    check(a, st, one + [(0.2, word(n, {3: "Y", n - 1: "Z"}))])
    # two masks that share no tile: 8 flips above the low qubits each, disjoint
    apart = [(0.5, word(n, {q: "X" for q in range(4, 12)})), (0.4, word(n, {q: "X" for q in range(12, 20)}))]
    check(a, st, apart)
    check(a, st, apart + one + [(1.0, word(n, {0: "Z"}))])


def test_more_masks_than_the_window():
    n = 13
    r = np.random.default_rng(13)
    a, st = state(n, r)
    terms = [(float(r.normal()), "".join(r.choice(list("IXYZ"), n))) for _ in range(2500)]
    check(a, st, terms)
