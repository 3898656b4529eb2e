"""ket_batch_vqe's CTAs of 128, 256 and 512 threads and its packs against the oracle:
tiles of up to 2^13 amplitudes, one instance a CTA while all run at once, packs of up
to 32 where they do not, a template that no other shares its width with, and one that
no instance uses."""
import math

import numpy as np
import pytest

import ket_b200 as K
from ket_b200.batch import batch_vqe

pytestmark = pytest.mark.gpu

ANGLE = ("ry", "rz", "rx", "u1", "crx", "xx", "xy")


def template(n, depth, seed):
    """An ansatz, its Hamiltonian, and the same circuit on the oracle."""
    from oracle import oracle as O
    r = np.random.default_rng(seed)
    plan = []
    for _ in range(depth):
        k = str(r.choice(["ry", "rz", "rx", "h", "t", "u1", "cnot", "cnot", "swap", "crx", "cz", "xx", "xy", "ccx", "cswap"]))
        need = {"ccx": 3, "cswap": 3}.get(k, 2 if k in ("cnot", "swap", "crx", "cz", "xx", "xy") else 1)
        if need <= n:
            plan.append((k, [int(q) for q in r.permutation(n)[:need]]))

    def ansatz(p):
        c, i = K.Circuit(n), 0
        for k, q in plan:
            c = getattr(c, k)(*([p[i % len(p)]] if k in ANGLE else []), *q)
            i += k in ANGLE
        return c

    def oracle(p):
        c, i = O.OCircuit(n), 0
        for k, q in plan:
            c.add(k, q, [float(p[i % len(p)])] if k in ANGLE else [])
            i += k in ANGLE
        return c

    terms = [(float(r.normal()), "".join(r.choice(list("IXYZ"), n))) for _ in range(6)]
    terms += [(float(r.normal()), "".join(r.choice(list("IZ"), n))) for _ in range(4)]
    return ansatz, terms, oracle


def energy(state, terms):
    """sum_t c_t <P_t> on a dense state.  (The oracle's own vqe() simulates once more per
    term with the basis change, and flushes after that as well.)"""
    n = int(state.size).bit_length() - 1
    x = np.arange(state.size)
    total = 0.0
    for c, ops in terms:
        flip, sign, ny = 0, np.zeros(state.size, dtype=np.int64), 0
        for q in range(n):
            ch = ops[n - 1 - q]
            flip |= (ch in "XY") << q
            if ch in "YZ":
                sign ^= (x >> q) & 1
            ny += ch == "Y"
        total += c * float(np.real(1j ** ny * np.sum(np.conj(state[x ^ flip]) * (1 - 2 * sign) * state)))
    return total


@pytest.mark.parametrize("sizes,ninst,depth", [((1,), 1, 12), ((3,), 591, 20), ((3,), 593, 20), ((4,), 20000, 20), ((8,), 150, 60),
                                               ((8,), 2000, 60), ((10, 11), 400, 60), ((12,), 297, 60), ((13,), 149, 60),
                                               ((2, 13), 200, 60), ((5, 12), 900, 60)])
def test_against_the_oracle(sizes, ninst, depth):
    from oracle import oracle as O
    T = [template(n, depth, 100 * n + depth) for n in sizes]
    unused = (lambda p: K.Circuit(6).ry(p[0], 0), [(1.0, "Z" * 6)])
    r = np.random.default_rng(ninst)
    inst = [(i % len(sizes), r.uniform(0, 2 * math.pi, 5)) for i in range(ninst)]
    got = batch_vqe([t[:2] for t in T] + [unused], inst)
    assert got.shape == (ninst,)
    for i in {0, ninst - 1, ninst // 2, *[int(x) for x in r.integers(0, ninst, 5)]}:
        _, terms, oracle = T[inst[i][0]]
        want = energy(oracle(inst[i][1]).simulate(mode=O.DENSE_PRUNE).dense(), terms)
        # FP64 rounding of `depth` gates and their terms, and of merged diagonal factors
        assert abs(got[i] - want) <= 1e-14 * depth * sum(abs(c) for c, _ in terms), i


@pytest.mark.parametrize("n", [1, 3, 5, 6, 8, 9, 10, 11, 12, 13])
@pytest.mark.parametrize("ninst,strings", [(1, 1), (3, 37), (160, 90), (700, 20)])
def test_shares_of_the_hamiltonian(n, ninst, strings):
    """Threads beyond an instance's amplitudes take a share of its flip groups: fewer groups
    than shares, more, and packs."""
    from oracle import oracle as O
    ansatz, _, oracle = template(n, 20, 7 * n)
    r = np.random.default_rng(n + ninst)
    terms = [(float(r.normal()), "".join(r.choice(list("IXYZ"), n))) for _ in range(strings)]
    inst = [(0, r.uniform(0, 2 * math.pi, 5)) for _ in range(ninst)]
    got = batch_vqe([(ansatz, terms)], inst)
    ident = sum(c for c, o in terms if set(o) == {"I"})
    rest = [(c, o) for c, o in terms if set(o) != {"I"}]
    for i in {0, ninst - 1, ninst // 2}:
        want = ident + energy(oracle(inst[i][1]).simulate(mode=O.DENSE_PRUNE).dense(), rest)
        # FP64 rounding of 20 gates and the terms
        assert abs(got[i] - want) <= 2e-13 * sum(abs(c) for c, _ in terms)
