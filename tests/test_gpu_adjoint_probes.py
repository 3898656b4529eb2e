"""Probe forms of the compiled adjoint passes: Ry, Rx, Rz and U1 (whose
derivative matrices are taken in their own forms), controlled and general gates
beside them, targets in every register, lane and out-of-tile position, and passes
with up to and more than the 24 probes that keep a sum a thread.

Against the engine's parameter shift, which shares none of it: a gradient entry
is a quadratic form bounded by the sum S of the Hamiltonian's |coefficients|, and
each of the circuit's G gates rounds an amplitude at most 4 times (2^-53 each) in
psi and in lambda, forward and back; the two shifted energies likewise:
|difference| <= 32 G S 2^-53.  Controlled gates (no two-point shift rule):
central differences with eps = 1e-6, error 1e-7 as everywhere for them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ham(n):
    z = [(0.5 + 0.1 * q, "I" * q + "ZZ" + "I" * (n - q - 2)) for q in range(n - 1)]
    x = [(0.3 + 0.05 * q, "I" * q + "X" + "I" * (n - q - 1)) for q in range(n)]
    return z + x + [(0.4, ("XYZ" * n)[:n])]


def _ansatz(n, layers, kinds):
    """A layer puts each gate of `kinds` on every qubit, then a ring of CNOTs."""
    import ket_b200 as K

    def ans(p):
        c, k = K.Circuit(n), 0
        for _ in range(layers):
            for g in kinds:
                for q in range(n):
                    c = getattr(c, g)(p[k], q)
                    k += 1
            for q in range(n):
                c = c.cnot(q, (q + 1) % n)
        return c

    ans.paramCount = layers * len(kinds) * n
    ans.gates = layers * (len(kinds) + 1) * n
    return ans


@pytest.mark.parametrize("n,layers,kinds", [
    (12, 2, ("ry", "rz")),
    (13, 2, ("rx", "ry")),
    (12, 1, ("ry", "rz", "u1", "rz")),  # more than 24 diagonal probes in one pass
    (14, 1, ("ry", "rx", "u1")),
    (17, 1, ("rz", "rx")),
])
def test_rotation_probes_match_the_parameter_shift(n, layers, kinds):
    from ket_b200.adjoint import adjoint_gradient, shift_gradient
    ans, H = _ansatz(n, layers, kinds), _ham(n)
    P = np.random.default_rng(n).uniform(0, 2 * np.pi, size=(8, ans.paramCount))  # 8 vectors: compiled passes
    _, g = adjoint_gradient(ans, H, P)
    bound = 32 * ans.gates * sum(abs(c) for c, _ in H) * 2.0 ** -53
    for b in (0, 7):
        want = np.asarray(shift_gradient(ans, H, [list(P[b])])[1])[0]
        assert np.max(np.abs(g[b] - want)) <= bound


def test_controlled_and_general_probes_beside_them():
    import ket_b200 as K
    from ket_b200.adjoint import adjoint_gradient
    n = 14

    def ans(p):
        c = K.Circuit(n)
        for q in range(n):
            c = c.h(q)
        c = c.crx(p[0], 0, 5).cry(p[1], 13, 1).crz(p[2], 11, 3).cu1(p[3], 2, 12).crz(p[4], 4, 0).cry(p[5], 1, 2)
        return c.gpi(p[6], 5).gpi2(p[7], 13).ry(p[8], 9).rz(p[9], 9).xx(p[10], 1, 7).zz(p[11], 3, 10)

    H = _ham(n)
    P = np.random.default_rng(5).uniform(0, 2 * np.pi, size=(8, 12))
    _, g = adjoint_gradient(ans, H, P)
    eps = 1e-6
    for k in range(12):
        hi, lo = list(P[3]), list(P[3])
        hi[k] += eps
        lo[k] -= eps
        assert abs((K.vqe(ans(hi), H) - K.vqe(ans(lo), H)) / (2 * eps) - g[3, k]) < 1e-7
