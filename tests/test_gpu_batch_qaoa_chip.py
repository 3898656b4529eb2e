"""Batched QAOA instances that fit the chip run apart from the wide ones: batches of
either kind alone and of both, narrow batches of more instances than the grid holds,
replayed graphs of alternating shapes, and p = 0, against a dense simulation."""
import numpy as np
import pytest

from ket_b200 import _lib, autotune
from ket_b200.batch import batch_qaoa
from test_gpu_batch_qaoa_tiles import dense_cut, instances

pytestmark = pytest.mark.gpu


def check(inst, got):
    for (n, e, g, b), v in zip(inst, got):
        # a few hundred FP64 roundings an amplitude, <C> of order |E|
        assert abs(v - dense_cut(n, e, g, b)) <= 1e-12 * max(1, len(e)), n


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("sizes", [[1], [2, 3], [12], [13], [14, 12, 13, 1], list(range(1, 13))])
def test_kinds_of_batches(sizes, graph):
    for p in (1, 3):
        inst = instances(sizes, p, 7 * len(sizes) + p)
        check(inst, batch_qaoa(inst, use_graph=graph))


def test_alternating_shapes_replay_their_own_graphs():
    batches = [instances(sizes, 2, k) for k, sizes in enumerate(([3, 4], [13, 4], [13], [3, 4], [12, 14, 2]))]
    for _ in range(2):
        for inst in batches:
            check(inst, batch_qaoa(inst))
            check(inst, batch_qaoa(inst))


@pytest.mark.parametrize("threads", [128, 256, 512])
def test_more_instances_than_ctas(threads):
    inst = instances([2, 5, 3, 6] * 1000, 2, 11)
    autotune.set_batch_config(threads, 0)
    try:
        got = batch_qaoa(inst)
    finally:
        autotune.set_batch_config(0, 0)
    check(inst[:40], got)
    for k in (1999, 3998, 3999):
        check(inst[k:k + 1], got[k:k + 1])
    assert np.array_equal(got, batch_qaoa(inst)) or threads != 256


def test_no_layers_beside_any_width():
    edges = [(0, 1), (1, 2)]
    got = batch_qaoa([(24, edges, [], []), (3, edges, [], []), (1, [], [], [])])
    assert got.tolist() == [1.0, 1.0, 0.0]


def test_narrow_batch_is_one_launch():
    """No phase tables, tiles or reduction where every instance fits the chip."""
    import ctypes as C
    count = C.c_uint64()
    def launches():
        _lib.check(_lib.lib().ket_ctx_launch_count(_lib.default_ctx(), C.byref(count)))
        return count.value
    inst = instances([4, 9, 12], 2, 3)
    batch_qaoa(inst)
    at = launches()
    batch_qaoa(inst)
    assert launches() - at == 1


def test_rounding_does_not_build_up():
    """<C> over the norm: the rounding of one cosine and sine, the same in every rotation of
    a layer, must not add up over qubits and layers."""
    inst = []
    r = np.random.default_rng(4)
    for _ in range(60):
        n = 9
        edges = [(i, (i + 1) % n) for i in range(n)] + [(0, 3), (1, 5)]
        inst.append((n, edges, r.uniform(0, 3, 8).tolist(), r.uniform(0, 1.5, 8).tolist()))
    got = batch_qaoa(inst)
    worst = 0.0
    for (n, edges, gamma, beta), v in zip(inst, got):
        x = np.arange(1 << n)
        cut = np.zeros(1 << n, dtype=np.longdouble)
        for u, w in edges:
            cut += ((x >> u) ^ (x >> w)) & 1
        a = np.full(1 << n, 1 / np.sqrt(np.longdouble(1 << n)), dtype=np.clongdouble)
        for g, b in zip(gamma, beta):
            a = a * np.exp(-1j * (np.longdouble(g) * (len(edges) - 2 * cut)).astype(np.clongdouble))
            c, s = np.cos(np.longdouble(b)), np.sin(np.longdouble(b))
            for q in range(n):
                y = a.reshape(-1, 2, 1 << q)
                y0, y1 = y[:, 0].copy(), y[:, 1].copy()
                y[:, 0], y[:, 1] = c * y0 - 1j * s * y1, c * y1 - 1j * s * y0
        worst = max(worst, float(abs(v - ((a.real ** 2 + a.imag ** 2) * cut).sum())))
    # <C> of up to 11: an ulp of it is 1.8e-15.  Sums over 512 products and the quotient round
    # a few times; without the norm, 2 x 72 rotations a state shift it by up to 144 x 2^-53 x 11
    assert worst <= 4 * 1.8e-15
