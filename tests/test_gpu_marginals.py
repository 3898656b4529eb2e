"""Marginals and joint distributions against numpy: states below, at and above
one 2^12 block, with the joint's qubits on thread, register, loop and block bits."""
import numpy as np
import pytest

from ket_b200.circuit import DeviceState, KET_C64, KET_C128

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [KET_C128, KET_C64])
@pytest.mark.parametrize("n", [1, 4, 11, 12, 13, 18, 23, 25])
def test_marginals_and_joint(n, precision):
    r = np.random.default_rng(n)
    a = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    a /= np.linalg.norm(a)
    if precision == KET_C64:
        a = a.astype(np.complex64).astype(np.complex128)
    st = DeviceState(n, precision)
    st.set_amplitudes(a)
    p = a.real ** 2 + a.imag ** 2
    # sums of at most 2^25 positive terms that add up to 1, in runs of a few hundred: under 1e3 roundings
    want = [p.reshape(-1, 2, 1 << q)[:, 1].sum() for q in range(n)]
    assert np.abs(st.marginals() - want).max() <= 1e-13
    sets = [[0], [n - 1], list(range(min(n, 12))), list(range(n - 1, max(-1, n - 13), -1))]
    sets += [[int(q) for q in r.permutation(n)[:m]] for m in (1, 3, 7, 12) if m <= n]
    for qs in sets:
        axes = [n - 1 - q for q in reversed(qs)]
        v = p.reshape([2] * n).transpose(axes + [i for i in range(n) if i not in axes])
        assert np.abs(st.marginal_dist(qs) - v.reshape(1 << len(qs), -1).sum(1)).max() <= 1e-13
