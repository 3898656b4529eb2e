"""The batched QAOA's passes and layouts against a dense simulation: instances
below, at and above one tile, both tile widths on every CTA size, odd and even
layer counts, repeated edges, no edges, angles around pi/2, and p = 0."""
import math

import numpy as np
import pytest

from ket_b200 import autotune
from ket_b200.batch import batch_qaoa

pytestmark = pytest.mark.gpu


def dense_cut(n, edges, gamma, beta):
    x = np.arange(1 << n)
    cut = np.zeros(1 << n)
    for u, v in edges:
        cut += ((x >> u) ^ (x >> v)) & 1
    a = np.full(1 << n, 2.0 ** (-n / 2), dtype=complex)
    for g, b in zip(gamma, beta):
        a = a * np.exp(-1j * g * (len(edges) - 2 * cut))
        for q in range(n):
            v = a.reshape(-1, 2, 1 << q)
            v0, v1 = v[:, 0].copy(), v[:, 1].copy()
            v[:, 0], v[:, 1] = math.cos(b) * v0 - 1j * math.sin(b) * v1, math.cos(b) * v1 - 1j * math.sin(b) * v0
    return float(np.sum(np.abs(a) ** 2 * cut))


def instances(sizes, p, seed):
    r = np.random.default_rng(seed)
    out = []
    for n in sizes:
        every = [(u, v) for u in range(n) for v in range(u + 1, n)]
        m = int(min(64, len(every), r.integers(0, 2 * n + 1)))
        edges = [every[i] if r.random() < 0.5 else every[i][::-1] for i in r.permutation(len(every))[:m]]
        if edges and r.random() < 0.4 and len(edges) < 64:
            edges.append(edges[0][::-1])  # the same edge again
        gamma = r.uniform(0, math.pi, p).tolist()
        beta = [float(r.choice([math.pi / 2, -math.pi / 2, math.pi / 4, 0.0, b])) for b in r.uniform(-4, 4, p)]
        out.append((n, edges, gamma, beta))
    return out


@pytest.mark.parametrize("p", [1, 2, 3, 6])
@pytest.mark.parametrize("threads,tile", [(128, 11), (256, 11), (512, 11), (128, 12), (256, 12), (512, 12)])
def test_qaoa_tiles(threads, tile, p):
    inst = instances([1, 2, 3, 4, 5, 8, 9, 10, 11, 12, 12, 13, 13, 14, 15, 16], p, 10 * p + threads + tile)
    autotune.set_batch_config(threads, tile)
    try:
        got = batch_qaoa(inst)
    finally:
        autotune.set_batch_config(0, 0)
    for (n, e, g, b), v in zip(inst, got):
        # a few hundred FP64 roundings an amplitude, <C> of order |E|
        assert abs(v - dense_cut(n, e, g, b)) <= 1e-12 * max(1, len(e)), (n, p)


def test_qaoa_widest_and_no_layers():
    inst = instances([19, 22], 2, 3)
    for (n, e, g, b), v in zip(inst, batch_qaoa(inst)):
        assert abs(v - dense_cut(n, e, g, b)) <= 1e-12 * max(1, len(e))
    edges = [(0, 1), (1, 2), (5, 23)]
    assert np.allclose(batch_qaoa([(24, edges, [], []), (3, edges[:2], [], [])]), [1.5, 1.0], rtol=0, atol=1e-15)
