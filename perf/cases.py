"""The work a user has the engine do, as a list of timed cases.

Each case names one call, or the few calls of one step, of a program that uses
the engine: simulating a circuit and reading it out (on a resident DeviceState,
as a program that simulates again and again holds one), the read-outs of a large
state, adjoint gradients, batches of variational circuits, noisy per-shot runs
and density matrices.  Sizes run from a few qubits to the 30-qubit state of the
benchmark.  A case fixes the structure of a circuit; the seed of prepare() gives
its angles, basis states, graphs, parameters and draws.

exact() restates the same computations with torch in complex128, with the
reference's pruning of every computed amplitude with |a|^2 < 1e-14.
"""
import math
import random

import numpy as np
import torch

PRUNE = 1e-14


def listed():
    return [
        # the smallest call: a few qubits, the whole state read back (a unit test, an interactive session)
        {"name": "state_10q", "kind": "circuit", "family": "brick", "n": 10, "layers": 10, "structure": 1,
         "precision": "c128", "prune": True, "compiled": False, "read": "state"},
        # the reference's own size: simulate, exact probabilities, 4096 shots
        {"name": "shots_16q", "kind": "circuit", "family": "brick", "n": 16, "layers": 20, "structure": 42,
         "precision": "c128", "prune": True, "compiled": False, "read": "shots"},
        # the largest circuit of the reference's published benchmark, the Fourier transform of a basis state
        {"name": "qft_20q", "kind": "circuit", "family": "qft", "n": 20, "layers": 1, "structure": 1,
         "precision": "c128", "prune": True, "compiled": False, "read": "amplitudes"},
        # every kind of gate, an odd size, single precision, no pruning, kernels compiled ahead of the first run
        {"name": "mixed_25q_c64", "kind": "circuit", "family": "mixed", "n": 25, "layers": 6, "structure": 7,
         "precision": "c64", "prune": False, "compiled": True, "read": "amplitudes"},
        # the benchmark's step: a 16 GiB state, 40 layers and a Fourier transform
        {"name": "step_30q", "kind": "circuit", "family": "brick_qft", "n": 30, "layers": 40, "structure": 42,
         "precision": "c128", "prune": True, "compiled": True, "read": "amplitudes"},
        # the read-outs of one large resident state: marginals, a joint distribution, an energy, shots
        {"name": "readout_27q", "kind": "readout", "n": 27, "precision": "c128", "joint": 10, "shots": 4096},
        # one step of a small variational optimisation
        {"name": "gradient_14q", "kind": "gradient", "n": 14, "layers": 3, "vectors": 1},
        # gradients of the 24-qubit, 8-layer ansatz for a batch of parameter vectors
        {"name": "gradient_24q", "kind": "gradient", "n": 24, "layers": 8, "vectors": 8},
        # QAOA instances of uneven width in one call
        {"name": "qaoa_512", "kind": "qaoa", "instances": 512, "low": 10, "high": 22, "regular": True, "p": 4},
        # a parameter sweep of variational energies over circuits of uneven width
        {"name": "vqe_2048", "kind": "vqe", "instances": 2048, "low": 8, "high": 13, "layers": 4},
        # noisy shots of a circuit with a measurement and a reset in it
        {"name": "noisy_12q", "kind": "noisy", "n": 12, "layers": 8, "structure": 9, "shots": 16384},
        # the exact density matrix of a noisy circuit
        {"name": "density_11q", "kind": "density", "n": 11, "layers": 4, "structure": 5},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["circuit", "circuit", "circuit", "readout", "gradient", "qaoa", "vqe", "noisy", "density"])
    if kind == "circuit":
        n = rng.randint(3, 27)
        family = rng.choice(["brick", "brick_qft", "mixed", "qft"])
        return {"kind": kind, "family": family, "n": n, "layers": rng.randint(2, 24 if n < 24 else 8),
                "structure": rng.randint(1, 1 << 20), "precision": rng.choice(["c128", "c128", "c64"]),
                "prune": rng.random() < 0.7, "compiled": n >= 26 or (n >= 14 and rng.random() < 0.3),
                "read": "state" if n <= 12 else rng.choice(["shots", "amplitudes"]) if n <= 18 else "amplitudes"}
    if kind == "readout":
        n = rng.randint(14, 28)
        return {"kind": kind, "n": n, "precision": rng.choice(["c128", "c64"]), "joint": rng.randint(1, 12),
                "shots": _log_int(rng, 16, 1 << 15)}
    if kind == "gradient":
        n = rng.randint(5, 23)
        return {"kind": kind, "n": n, "layers": rng.randint(1, 8), "vectors": _log_int(rng, 1, 12)}
    if kind == "qaoa":
        low = rng.randint(4, 18)
        return {"kind": kind, "instances": _log_int(rng, 4, 512 if low < 14 else 96), "low": low, "high": low + rng.randint(0, 4),
                "regular": rng.random() < 0.4, "p": rng.randint(1, 6)}
    if kind == "vqe":
        low = rng.randint(3, 13)
        return {"kind": kind, "instances": _log_int(rng, 4, 4096), "low": low, "high": rng.randint(low, 13),
                "layers": rng.randint(1, 6)}
    if kind == "noisy":
        return {"kind": kind, "n": rng.randint(2, 12), "layers": rng.randint(1, 12), "structure": rng.randint(1, 1 << 20),
                "shots": _log_int(rng, 16, 16384)}
    return {"kind": kind, "n": rng.randint(3, 11), "layers": rng.randint(1, 5), "structure": rng.randint(1, 1 << 20)}


# ---------------------------------------------------------------- circuits as plain gate lists
# A gate is (name, params, qubits), or ("unitary", matrix, qubits).


def _brick(n, layers, kinds, ang):
    """Layers of one H, T, Rx, Ry or Rz a qubit, then CNOTs between neighbours."""
    gates = []
    for l in range(layers):
        for q in range(n):
            g = kinds.choice(["h", "t", "rx", "ry", "rz"])
            gates.append((g, [] if g in ("h", "t") else [ang.uniform(0, 2 * math.pi)], [q]))
        gates += [("cnot", [], [q, q + 1]) for q in range(l & 1, n - 1, 2)]
    return gates


def _qft(n):
    gates = []
    for j in range(n - 1, -1, -1):
        gates.append(("h", [], [j]))
        gates += [("cu1", [math.pi / 2 ** (j - k)], [k, j]) for k in range(j - 1, -1, -1)]
    return gates + [("swap", [], [i, n - 1 - i]) for i in range(n // 2)]


def _unitary3(ang):
    g = np.array([[complex(ang.gauss(0, 1), ang.gauss(0, 1)) for _ in range(8)] for _ in range(8)])
    return np.linalg.qr(g)[0]


def _mixed(n, layers, kinds, ang):
    """Layers of u3 on every qubit, then two- and three-qubit gates of every kind on random qubits."""
    gates = []
    for _ in range(layers):
        for q in range(n):
            gates.append(("u3", [ang.uniform(0, math.pi), ang.uniform(0, 6.28), ang.uniform(0, 6.28)], [q]))
        for _ in range(max(1, n // 3)):
            g = kinds.choice(["cnot", "cu1", "crx", "cry", "cz", "swap", "xx", "zz", "ccx", "cswap", "unitary"])
            k = 3 if g in ("ccx", "cswap", "unitary") else 2
            qs = kinds.sample(range(n), k)
            if g == "unitary":
                gates.append((g, _unitary3(ang), qs))
            else:
                gates.append((g, [ang.uniform(0, 2 * math.pi)] if g in ("cu1", "crx", "cry", "xx", "zz") else [], qs))
    return gates


def _circuit(case, seed):
    """(gate list, index of the basis state it starts from)"""
    kinds, ang = random.Random(case["structure"]), random.Random(seed)
    n, family = case["n"], case["family"]
    init = ang.randrange(1 << n)
    if family == "qft":
        return _qft(n), init
    if family == "mixed":
        return _mixed(n, case["layers"], kinds, ang), 0
    return _brick(n, case["layers"], kinds, ang) + (_qft(n) if family == "brick_qft" else []), 0


def _build(n, gates):
    from ket_b200.circuit import Circuit
    c = Circuit(n)
    for name, params, qs in gates:
        if name == "unitary":
            c = c.unitary([[complex(v) for v in row] for row in params], *qs)
        else:
            c = getattr(c, name)(*params, *qs)
    return c


def _amp_indices(n, seed):
    return np.random.default_rng(seed).integers(0, 1 << n, size=min(1024, 1 << n)).astype(np.uint64)


def _joint_qubits(n, m, seed):
    return random.Random(seed).sample(range(n), min(m, n))


def _tfim(n, seed):
    """-sum Z_i Z_(i+1) - sum h_i X_i; the first character of a term acts on the top qubit."""
    r, terms = random.Random(seed), []
    for i in range(n - 1):
        terms.append((-1.0, "".join("Z" if q in (i, i + 1) else "I" for q in reversed(range(n)))))
    for i in range(n):
        terms.append((-r.uniform(0.5, 1.5), "".join("X" if q == i else "I" for q in reversed(range(n)))))
    return terms


def _ansatz(n, layers):
    """Layers of Ry and Rz on every qubit and a ladder of CNOTs."""
    from ket_b200.workloads import hea_ladder
    return hea_ladder(n, layers)


def _graph(n, regular, r):
    if regular and n % 2 == 0 and n >= 4:
        while True:
            p = [i // 3 for i in range(3 * n)]
            r.shuffle(p)
            e = {(min(p[i], p[i + 1]), max(p[i], p[i + 1])) for i in range(0, 3 * n, 2)}
            if len(e) == 3 * n // 2 and all(u != v for u, v in e):
                return sorted(e)
    every = [(u, v) for u in range(n) for v in range(u + 1, n)]
    return r.sample(every, min(len(every), 3 * n // 2, 64))


def _qaoa_instances(case, seed):
    r, out = random.Random(seed), []
    for _ in range(case["instances"]):
        n = r.randrange(case["low"], case["high"] + 1, 2 if case["regular"] else 1)
        out.append((n, _graph(n, case["regular"], r), [r.uniform(0, math.pi) for _ in range(case["p"])],
                    [r.uniform(0, math.pi) for _ in range(case["p"])]))
    return out


def _vqe_instances(case, seed):
    sizes = range(case["low"], case["high"] + 1)
    r = np.random.default_rng(seed)
    which = r.integers(0, len(sizes), case["instances"])
    return sizes, [(int(t), r.uniform(0, 2 * math.pi, 2 * sizes[t] * case["layers"])) for t in which]


# ---------------------------------------------------------------- the cases


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("circuit", "readout"):
        from ket_b200.circuit import DeviceState, KET_C64, KET_C128
        n = case["n"]
        precision = KET_C64 if case["precision"] == "c64" else KET_C128
        s["state"] = DeviceState(n, precision)
        s["draws"] = np.random.default_rng(seed).random(case.get("shots", 4096))
    if kind == "circuit":
        gates, s["init"] = _circuit(case, seed)
        c = _build(n, gates)
        s["abi"] = c.to_abi()
        if case["compiled"]:
            c.compile_kernels(precision, case["prune"])
        s["prune"], s["read"] = case["prune"], case["read"]
        s["indices"], s["joint"] = _amp_indices(n, seed), list(range(min(10, n)))
    elif kind == "readout":
        s["state"].apply_abi(*_build(n, _brick(n, 3, random.Random(1), random.Random(seed))).to_abi())
        s["joint"], s["terms"] = _joint_qubits(n, case["joint"], seed), _tfim(n, seed)
    elif kind == "gradient":
        s["ansatz"], s["terms"] = _ansatz(case["n"], case["layers"]), _tfim(case["n"], seed)
        s["params"] = np.random.default_rng(seed).uniform(0, 2 * math.pi, (case["vectors"], 2 * case["n"] * case["layers"]))
    elif kind == "qaoa":
        s["instances"] = _qaoa_instances(case, seed)
    elif kind == "vqe":
        sizes, s["instances"] = _vqe_instances(case, seed)
        s["templates"] = [(_ansatz(n, case["layers"]), _tfim(n, seed + n)) for n in sizes]
    else:
        kinds, ang = random.Random(case["structure"]), random.Random(seed)
        c = _build(case["n"], _brick(case["n"], case["layers"], kinds, ang))
        if kind == "noisy":
            c = c.creg("c", 1).measure(0, "c", 0).reset(0).append(_build(case["n"], _brick(case["n"], 2, kinds, ang)))
            s["shots"], s["seed"] = case["shots"], 1 + seed % (1 << 31)
        s["circuit"] = c
    return s


def run(s):
    kind = s["kind"]
    if kind == "circuit":
        st = s["state"]
        st.set_basis(s["init"])
        st.apply_abi(*s["abi"], prune=s["prune"])
        if s["read"] == "state":
            return {"state": st.amplitudes_dense()}
        if s["read"] == "shots":
            return {"probabilities": st.probs_dense(), "shots": st.sample(s["draws"])}
        return {"amplitudes": st.amplitudes(s["indices"]), "joint": st.marginal_dist(s["joint"])}
    if kind == "readout":
        st = s["state"]
        return {"marginals": st.marginals(), "joint": st.marginal_dist(s["joint"]),
                "energy": st.expect_pauli_sum(s["terms"]), "norm": st.norm2(), "shots": st.sample(s["draws"])}
    if kind == "gradient":
        from ket_b200.adjoint import adjoint_gradient
        energies, gradients = adjoint_gradient(s["ansatz"], s["terms"], s["params"])
        return {"energies": energies, "gradients": gradients}
    if kind == "qaoa":
        from ket_b200.batch import batch_qaoa
        return {"cuts": batch_qaoa(s["instances"])}
    if kind == "vqe":
        from ket_b200.batch import batch_vqe
        return {"energies": batch_vqe(s["templates"], s["instances"])}
    if kind == "noisy":
        indices, bits, _, stream = s["circuit"].run_shots(s["shots"], s["seed"], "aria-1")
        return {"indices": indices, "bits": bits, "stream": stream}
    rho = s["circuit"].dm("aria-1")
    diagonal = np.zeros(1 << rho.qubits)
    for key, p in rho.probabilities().items():
        diagonal[int(key[::-1], 2)] = p
    return {"probabilities": diagonal, "purity": rho.purity(), "theta": rho.blochAngles(0)["theta"]}


# ---------------------------------------------------------------- work


_FLOPS = {"h": 6, "rx": 6, "ry": 6, "rz": 6, "t": 3, "u3": 14, "cu1": 1.5, "cz": 0, "crx": 3, "cry": 3, "xx": 14,
          "zz": 6, "unitary": 62, "cnot": 0, "swap": 0, "ccx": 0, "cswap": 0}


def _flops(gates, n):
    """Real operations of the gates on 2^n amplitudes: 6 a complex product, 2 a sum, real factors counted as such."""
    return sum(_FLOPS[g[0]] for g in gates) * float(1 << n)


def work(case):
    """The state (or the pair of states a gradient carries) written once, the outputs, and the gates' arithmetic."""
    kind = case["kind"]
    if kind == "circuit":
        n, amp = case["n"], 8 if case["precision"] == "c64" else 16
        gates, _ = _circuit(case, 1)
        return {"bytes": amp * (1 << n) * (2 if case["read"] == "state" else 1) + 16 * 1024, "flops": _flops(gates, n)}
    if kind == "readout":
        n, amp = case["n"], 8 if case["precision"] == "c64" else 16
        return {"bytes": amp * (1 << n), "flops": (3 + n + 1 + 8 * n) * float(1 << n)}
    if kind == "gradient":
        n, p = case["n"], 2 * case["n"] * case["layers"]
        return {"bytes": case["vectors"] * 32 * (1 << n), "flops": case["vectors"] * (3 * 6 + 4) * p * float(1 << n)}
    if kind == "qaoa":
        inst = _qaoa_instances(case, 1)
        return {"bytes": 8 * case["instances"] * (2 * case["p"] + 1) + sum(8 * len(e) for _, e, _, _ in inst),
                "flops": sum((6 * n + 6) * case["p"] * float(1 << n) for n, _, _, _ in inst)}
    if kind == "vqe":
        sizes, inst = _vqe_instances(case, 1)
        return {"bytes": 8 * sum(len(p) + 1 for _, p in inst),
                "flops": sum((12 * sizes[t] * case["layers"] + 8 * sizes[t]) * float(1 << sizes[t]) for t, _ in inst)}
    n = case["n"]
    gates = _brick(n, case["layers"] + 2 * (kind == "noisy"), random.Random(case["structure"]), random.Random(1))
    if kind == "noisy":
        return {"bytes": 9.0 * case["shots"], "flops": case["shots"] * (_flops(gates, n) + 12.0 * (1 << n))}
    # on the row and on the column index, with a depolarising channel after each gate
    return {"bytes": 16 * (1 << 2 * n) + 8 * (1 << n), "flops": 2 * _flops(gates, 2 * n) + 8.0 * len(gates) * (1 << 2 * n)}


# ---------------------------------------------------------------- exact values


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _matrix(name, p):
    e = lambda a: complex(math.cos(a), math.sin(a))
    if name == "unitary":
        return np.asarray(p)
    c, s = (math.cos(p[0] / 2), math.sin(p[0] / 2)) if p else (0.0, 0.0)
    r = math.sqrt(0.5)
    return np.array({
        "h": lambda: [[r, r], [r, -r]], "t": lambda: [[1, 0], [0, e(math.pi / 4)]],
        "rx": lambda: [[c, -1j * s], [-1j * s, c]], "ry": lambda: [[c, -s], [s, c]],
        "rz": lambda: [[e(-p[0] / 2), 0], [0, e(p[0] / 2)]],
        "u3": lambda: [[c, -s * e(p[2])], [s * e(p[1]), c * e(p[1] + p[2])]],
        "cu1": lambda: [[1, 0], [0, e(p[0])]], "cz": lambda: [[1, 0], [0, -1]],
        "crx": lambda: [[c, -1j * s], [-1j * s, c]], "cry": lambda: [[c, -s], [s, c]],
        "xx": lambda: [[c, 0, 0, -1j * s], [0, c, -1j * s, 0], [0, -1j * s, c, 0], [-1j * s, 0, 0, c]],
        "zz": lambda: np.diag([e(-p[0] / 2), e(p[0] / 2), e(p[0] / 2), e(-p[0] / 2)]),
    }[name](), dtype=complex)


def _flush(a, prune):
    if prune:
        v = torch.view_as_real(a)
        v.mul_(((v * v).sum(-1, keepdim=True) >= PRUNE).to(v.dtype))


def _split(a, q):
    """`a` [..., 2^n] as [..., high, 2, low] around qubit q."""
    return a.view(*a.shape[:-1], -1, 2, 1 << q)


def _mat1(a, m, q, prune):
    """A 2x2 on qubit q; an entry of m is a number or a tensor over the batch."""
    v = _split(a, q)
    x0, x1 = v[..., 0, :].clone(), v[..., 1, :]
    y1 = m[1][0] * x0 + m[1][1] * x1
    v[..., 0, :] = m[0][0] * x0 + m[0][1] * x1
    v[..., 1, :] = y1
    _flush(a, prune)


def _matk(a, m, qs, prune):
    """A 2^k x 2^k on qubits qs of a flat state, the first of them the top bit of its index."""
    n = a.numel().bit_length() - 1
    axes = [n - 1 - q for q in qs]
    v = a.view([2] * n).movedim(axes, list(range(len(qs))))
    y = torch.as_tensor(m, dtype=a.dtype, device=a.device) @ v.reshape(1 << len(qs), -1)
    v.copy_(y.view([2] * n))
    _flush(a, prune)


def _exact_gate(a, gate, prune):
    name, p, qs = gate
    n = a.shape[-1].bit_length() - 1
    if name in ("h", "t", "rx", "ry", "rz", "u3"):
        _mat1(a, _matrix(name, p).tolist(), qs[0], prune)
    elif name in ("xx", "zz", "unitary"):
        _matk(a, _matrix(name, p), qs, prune)
    else:
        v = a.view([2] * n)
        ctl = {"ccx": 2}.get(name, 0 if name == "swap" else 1)
        at = [slice(None)] * n
        for q in qs[:ctl]:
            at[n - 1 - q] = 1
        if name in ("swap", "cswap"):
            x, y = list(at), list(at)
            x[n - 1 - qs[-2]], x[n - 1 - qs[-1]] = 1, 0
            y[n - 1 - qs[-2]], y[n - 1 - qs[-1]] = 0, 1
        else:
            x, y = list(at), list(at)
            x[n - 1 - qs[-1]], y[n - 1 - qs[-1]] = 0, 1
        x, y = tuple(x), tuple(y)
        x0, x1 = v[x].clone(), v[y].clone()
        if name in ("cnot", "ccx", "swap", "cswap"):
            v[x], v[y] = x1, x0
        else:
            m = _matrix(name, p)
            v[x] = complex(m[0, 0]) * x0 + complex(m[0, 1]) * x1
            v[y] = complex(m[1, 0]) * x0 + complex(m[1, 1]) * x1
            _flush(a, prune)


def _exact_state(n, gates, init, prune):
    a = torch.zeros(1 << n, dtype=torch.complex128, device=_device())
    a[init] = 1
    for g in gates:
        _exact_gate(a, g, prune)
    return a


def _exact_joint(p, n, qubits):
    """Distribution of `qubits`, bit k of a bin = qubits[k]."""
    keep = [n - 1 - q for q in reversed(qubits)]
    v = p.view([2] * n).permute(keep + [i for i in range(n) if i not in keep])
    return v.reshape(1 << len(qubits), -1).sum(1)


def _abs2(a):
    v = torch.view_as_real(a)
    return (v * v).sum(-1)


def _hamiltonian(a, terms):
    """sum of terms of Z and X strings applied to states a [..., 2^n]"""
    n = a.shape[-1].bit_length() - 1
    idx = torch.arange(1 << n, device=a.device)
    d, out = torch.zeros(1 << n, dtype=torch.float64, device=a.device), torch.zeros_like(a)
    for c, t in terms:
        ops = t[::-1]
        if "X" in t:
            q = ops.index("X")
            out += c * _split(a, q).flip(-2).reshape(a.shape)
        else:
            sign = torch.ones_like(d)
            for q in range(n):
                if ops[q] == "Z":
                    sign *= 1 - 2 * ((idx >> q) & 1)
            d += c * sign
    return out.add_(d * a)


def _dot(a, b):
    """Re <a|b> over the last axis"""
    return (torch.view_as_real(a) * torch.view_as_real(b)).sum((-1, -2))


def _cnot(a, c, t):
    n = a.shape[-1].bit_length() - 1
    lo, hi = min(c, t), max(c, t)
    v = a.view(*a.shape[:-1], 1 << (n - 1 - hi), 2, 1 << (hi - lo - 1), 2, 1 << lo)
    x, y = (v[..., 1, :, 0, :], v[..., 1, :, 1, :]) if c == hi else (v[..., 0, :, 1, :], v[..., 1, :, 1, :])
    keep = x.clone()
    x.copy_(y)
    y.copy_(keep)


def _ladder_gate(a, g, angle, prune=False):
    """A gate of the ansatz at an angle (a number, or a column over the batch)."""
    name, q = g[0], g[1]
    if name == "cnot":
        return _cnot(a, q, q + 1)
    half = torch.as_tensor(angle, dtype=torch.float64, device=a.device) / 2
    c, s = torch.cos(half), torch.sin(half)
    if half.dim():
        c, s = c.view(-1, 1, 1), s.view(-1, 1, 1)
    if name == "ry":
        _mat1(a, [[c, -s], [s, c]], q, prune)
    else:
        v = _split(a, q)
        v[..., 0, :] *= torch.complex(c, -s)
        v[..., 1, :] *= torch.complex(c, s)
        _flush(a, prune)


def _ladder(n, layers):
    gates, k = [], 0
    for _ in range(layers):
        for q in range(n):
            gates += [("ry", q, k), ("rz", q, k + 1)]
            k += 2
        gates += [("cnot", q, -1) for q in range(n - 1)]
    return gates


def _exact_gradient(n, layers, terms, params):
    gates = _ladder(n, layers)
    psi = torch.zeros(1 << n, dtype=torch.complex128, device=_device())
    psi[0] = 1
    for g in gates:
        _ladder_gate(psi, g, params[g[2]] if g[2] >= 0 else 0.0)
    lam = _hamiltonian(psi, terms)
    energy, grad = float(_dot(psi, lam)), np.zeros(len(params))
    for g in reversed(gates):
        if g[2] >= 0:
            # d/dt exp(-i t G / 2) psi = -i/2 G psi after the gate
            p, l = _split(psi, g[1]), _split(lam, g[1])
            p0, p1, l0, l1 = p[..., 0, :], p[..., 1, :], l[..., 0, :], l[..., 1, :]
            if g[0] == "ry":  # -i/2 Y = [[0, -1/2], [1/2, 0]]
                d = _dot(l1, p0).sum() - _dot(l0, p1).sum()
            else:  # -i/2 Z
                d = torch.vdot(l0.reshape(-1), p0.reshape(-1)).imag - torch.vdot(l1.reshape(-1), p1.reshape(-1)).imag
            grad[g[2]] = float(d)
        angle = -params[g[2]] if g[2] >= 0 else 0.0
        _ladder_gate(psi, g, angle)
        _ladder_gate(lam, g, angle)
    return energy, grad


def _exact_cut(n, edges, gamma, beta):
    dev = _device()
    idx = torch.arange(1 << n, device=dev)
    cut = torch.zeros(1 << n, dtype=torch.float64, device=dev)
    for u, v in edges:
        cut += ((idx >> u) ^ (idx >> v)) & 1
    a = torch.full((1 << n,), 2.0 ** (-n / 2), dtype=torch.complex128, device=dev)
    for g, b in zip(gamma, beta):
        phase = -g * (len(edges) - 2 * cut)
        a *= torch.complex(torch.cos(phase), torch.sin(phase))
        c, s = math.cos(b), -1j * math.sin(b)
        k = min(n, 6)  # Rx on all qubits, six at a time as one 64 x 64
        for lo in range(0, n, k):
            m, w = np.array([[1.0 + 0j]]), min(k, n - lo)
            for _ in range(w):
                m = np.kron(m, np.array([[c, s], [s, c]]))
            v = a.view(-1, 1 << w, 1 << lo)
            a = torch.matmul(torch.as_tensor(m, device=dev), v).reshape(-1)
    return float((_abs2(a) * cut).sum())


def _exact_density(n, gates, p1, p2):
    """rho[row][col] as a state of 2n qubits, row bits on top; every op prunes its outputs once."""
    a = torch.zeros(1 << 2 * n, dtype=torch.complex128, device=_device())
    a[0] = 1
    x, z = np.array([[0, 1], [1, 0]], dtype=complex), np.diag([1.0 + 0j, -1])
    pauli = [np.eye(2, dtype=complex), x, 1j * x @ z, z]
    for name, p, qs in gates:
        if name == "cnot":
            c, t = qs
            _exact_gate(a, ("cnot", [], [n + c, n + t]), False)
            _exact_gate(a, ("cnot", [], [c, t]), False)
            ops, rate = [np.kron(u, v) for u in pauli for v in pauli][1:], p2
        else:
            m = _matrix(name, p)
            _matk(a, np.kron(m, m.conj()), [n + qs[0], qs[0]], True)
            ops, rate = pauli[1:], p1
        d = len(ops) + 1
        channel = (1 - rate) * np.eye(d, dtype=complex)
        for o in ops:
            channel += rate / (d - 1) * np.kron(o, o.conj())
        _matk(a, channel, [n + q for q in qs] + list(qs), True)
    return a.view(1 << n, 1 << n)


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "noisy":
        return None  # sampled indices and bits
    if kind == "circuit":
        if n > 27:
            return None  # more than a minute
        gates, init = _circuit(case, seed)
        a = _exact_state(n, gates, init, case["prune"])
        if case["read"] == "state":
            return {"state": a.cpu().numpy()}
        p = _abs2(a)
        if case["read"] == "shots":
            return {"probabilities": torch.where(p > PRUNE, p, 0).cpu().numpy(), "shots": None}
        at = torch.from_numpy(_amp_indices(n, seed).astype(np.int64)).to(a.device)
        return {"amplitudes": a[at].cpu().numpy(), "joint": _exact_joint(p, n, list(range(min(10, n)))).cpu().numpy()}
    if kind == "readout":
        a = _exact_state(n, _brick(n, 3, random.Random(1), random.Random(seed)), 0, True)
        p = _abs2(a)
        m = [float(_split(p, q)[:, 1].sum()) for q in range(n)]
        return {"marginals": np.array(m), "joint": _exact_joint(p, n, _joint_qubits(n, case["joint"], seed)).cpu().numpy(),
                "energy": float(_dot(a, _hamiltonian(a, _tfim(n, seed)))), "norm": float(p.sum()), "shots": None}
    if kind == "gradient":
        params = np.random.default_rng(seed).uniform(0, 2 * math.pi, (case["vectors"], 2 * n * case["layers"]))
        both = [_exact_gradient(n, case["layers"], _tfim(n, seed), [float(v) for v in p]) for p in params]
        return {"energies": np.array([e for e, _ in both]), "gradients": np.array([g for _, g in both])}
    if kind == "qaoa":
        return {"cuts": np.array([_exact_cut(*i) for i in _qaoa_instances(case, seed)])}
    if kind == "vqe":
        sizes, inst = _vqe_instances(case, seed)
        out = np.zeros(len(inst))
        for t, m in enumerate(sizes):
            mine = [i for i, (u, _) in enumerate(inst) if u == t]
            for first in range(0, len(mine), 256):
                some = mine[first:first + 256]
                a = torch.zeros((len(some), 1 << m), dtype=torch.complex128, device=_device())
                a[:, 0] = 1
                th = np.stack([inst[i][1] for i in some])
                for g in _ladder(m, case["layers"]):
                    _ladder_gate(a, g, th[:, g[2]] if g[2] >= 0 else 0.0, True)
                out[some] = _dot(a, _hamiltonian(a, _tfim(m, seed + m))).cpu().numpy()
        return {"energies": out}
    rho = _exact_density(n, _brick(n, case["layers"], random.Random(case["structure"]), random.Random(seed)), 0.0003, 0.005)
    v = _split(rho.diagonal().real, 0)
    z = float(v[:, 0].sum() - v[:, 1].sum())
    return {"probabilities": rho.diagonal().real.cpu().numpy(), "purity": float(_abs2(rho).sum()),
            "theta": math.acos(max(-1.0, min(1.0, z)))}
