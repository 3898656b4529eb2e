"""ket_batch_vqe's rounds, relabellings and packs against the engine's own
single-circuit vqe(): one to thirteen qubits, packs of one to 32 instances with a
short last one, runs of more matrices than shared memory holds at a time, gates
of every kind between relabellings, and terms that share flip masks."""
import math

import numpy as np
import pytest

import ket_b200 as K
from ket_b200.batch import batch_vqe

pytestmark = pytest.mark.gpu


def template(n, depth, seed):
    """A random circuit over every gate kind, its angles taken from the parameters in turn."""
    r = np.random.default_rng(seed)
    u2 = np.linalg.qr(r.normal(size=(4, 4)) + 1j * r.normal(size=(4, 4)))[0]
    plan = []
    for _ in range(depth):
        k = str(r.choice(["ry", "rz", "rx", "h", "t", "u1", "cnot", "cnot", "swap", "crx", "cz", "xx", "xy", "ccx", "cswap",
                          "csrswap", "u2"]))
        need = {"ccx": 3, "cswap": 3, "csrswap": 3}.get(k, 2 if k in ("cnot", "swap", "crx", "cz", "xx", "xy", "u2") else 1)
        if need <= n:
            plan.append((k, [int(q) for q in r.permutation(n)[:need]]))

    def ansatz(p):
        c, i = K.Circuit(n), 0
        for k, q in plan:
            if k in ("ry", "rz", "rx", "u1", "crx", "xx", "xy"):
                c = getattr(c, k)(p[i % len(p)], *q)
                i += 1
            elif k == "u2":
                c = c.unitary(u2, *q)
            else:
                c = getattr(c, k)(*q)
        return c

    terms = [(float(r.normal()), "".join(r.choice(list("IXYZ"), n))) for _ in range(2 * n)]
    terms += [(float(r.normal()), "".join(r.choice(list("IZ"), n))) for _ in range(6)]
    return ansatz, terms


@pytest.mark.parametrize("sizes,ninst,depth", [((1, 2, 3), 40, 20), ((4, 5), 300, 60), ((6, 8), 5000, 40), ((9, 10, 11), 700, 80),
                                               ((12, 13), 310, 90), ((7,), 4800, 150), ((13,), 3, 1200)])
def test_rounds_match_single_circuits(sizes, ninst, depth):
    templates = [template(n, depth, 10 * n + depth) for n in sizes]
    r = np.random.default_rng(ninst)
    inst = [(int(r.integers(len(sizes))), r.uniform(0, 2 * math.pi, 7)) for _ in range(ninst)]
    got = batch_vqe(templates, inst)
    for i in {0, 1, ninst - 1, *[int(x) for x in r.integers(0, ninst, 12)]}:
        t, p = inst[i]
        # FP64 rounding of `depth` gates and their terms, and of merged diagonal factors
        bound = 1e-14 * depth * sum(abs(c) for c, _ in templates[t][1])
        assert abs(got[i] - K.vqe(templates[t][0](p), templates[t][1])) <= bound, (i, sizes[t])
