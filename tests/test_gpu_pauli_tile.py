"""Pauli sums by tiles (12 and more qubits): flips inside and across passes,
flips too wide for a tile, groups below and above the direct-sign limit, Y
factors, and signs on thread, register and out-of-tile bits."""
import numpy as np
import pytest

from ket_b200.circuit import DeviceState, KET_C64, KET_C128

pytestmark = pytest.mark.gpu


def energy(a, terms):
    n = a.size.bit_length() - 1
    y = np.arange(a.size)
    e = 0.0
    for c, ops in terms:
        if set(ops) == {"I"}:  # an identity term adds its coefficient (algorithms.ts:310)
            e += c
            continue
        flip = sum(1 << q for q in range(n) if ops[n - 1 - q] in "XY")
        zm = sum(1 << q for q in range(n) if ops[n - 1 - q] in "YZ")
        par = np.zeros(a.size, dtype=np.int64)
        for q in range(n):
            if (zm >> q) & 1:
                par ^= (y >> q) & 1
        e += c * float(np.real(1j ** ops.count("Y") * np.sum((1 - 2 * par) * a * np.conj(a[y ^ flip]))))
    return e


def word(n, at):
    return "".join(at.get(q, "I") for q in reversed(range(n)))


@pytest.mark.parametrize("precision", [KET_C128, KET_C64])
@pytest.mark.parametrize("n", [11, 12, 13, 17, 21])
def test_pauli_sum_by_tiles(n, precision):
    r = np.random.default_rng(n)
    terms = [(float(r.normal()), word(n, {q: "X"})) for q in range(n)]
    terms += [(float(r.normal()), word(n, {q: "Z", q + 1: "Z"})) for q in range(n - 1)]
    for _ in range(24):  # any letters; flips wider than a tile from 17 qubits on
        terms.append((float(r.normal()), "".join(r.choice(list("IXYZ"), n))))
    for count in (1, 3, 4, 9):  # terms that share a flip mask
        f = [int(q) for q in r.permutation(n)[:2]]
        for _ in range(count):
            at = {q: "Z" for q in range(n) if q not in f and r.random() < 0.4}
            terms.append((float(r.normal()), word(n, {**at, **{q: str(r.choice(["X", "Y"])) for q in f}})))
    terms.append((0.7, "I" * n))
    a = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    a /= np.linalg.norm(a)
    if precision == KET_C64:
        a = a.astype(np.complex64).astype(np.complex128)
    st = DeviceState(n, precision)
    st.set_amplitudes(a)
    # FP64 products and sums of a unit vector: a few hundred roundings at most on any path to the result
    bound = 1e-13 * sum(abs(c) for c, _ in terms)
    assert abs(st.expect_pauli_sum(terms) - energy(a, terms)) <= bound
    for some in (terms[:1], terms[n - 1:n + 1], terms[-8:-4]):
        assert abs(st.expect_pauli_sum(some) - energy(a, some)) <= 1e-13 * sum(abs(c) for c, _ in some)


@pytest.mark.parametrize("n", [12, 15, 18])
def test_h_psi_by_tiles(n):
    """lambda = H psi in adjoint gradients: shared flip masks, Y factors and flips wider than a tile."""
    from ket_b200.adjoint import adjoint_gradient, shift_gradient
    from ket_b200.workloads import hea_ladder
    r = np.random.default_rng(50 + n)
    terms = [(float(r.normal()), word(n, {q: "X"})) for q in range(n)]
    terms += [(float(r.normal()), word(n, {q: "Z", q + 1: "Z"})) for q in range(n - 1)]
    terms += [(float(r.normal()), word(n, {0: a, n - 1: b, n // 2: c})) for a in "XY" for b in "XY" for c in "IZ"]
    terms += [(float(r.normal()), "".join(r.choice(list("IXYZ"), n))) for _ in range(6)]
    terms += [(float(r.normal()), "X" * n), (0.3, "I" * n)]
    ansatz = hea_ladder(n, 1)
    params = r.uniform(0, 6.28, (2, 2 * n))
    e, g = adjoint_gradient(ansatz, terms, params)
    es, gs = shift_gradient(ansatz, terms, params)
    # both are FP64 over a unit vector: a few thousand roundings at most, scaled by the terms' weights
    bound = 1e-12 * sum(abs(c) for c, _ in terms)
    assert np.abs(e - es).max() <= bound and np.abs(g - gs).max() <= bound
