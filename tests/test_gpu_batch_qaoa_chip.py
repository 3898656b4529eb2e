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
