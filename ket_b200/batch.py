"""Batched circuits in one persistent GPU launch, replayed from a CUDA graph:
QAOA MaxCut instances of uneven width (ket_batch_qaoa) and vqe() energies of
parameterised circuits of uneven width (ket_batch_vqe).

Instance i is (n, edges, gamma[p], beta[p]); the circuit is H on every qubit,
then per layer exp(-i gamma Z_u Z_v) on every edge and Rx(2 beta) on every
qubit, and the result is <C> = sum_edges (1 - <Z_u Z_v>)/2.  In the reference's
terms that is vqe(qaoa(n, edges, -2*gamma, beta), maxCutHamiltonian(n, edges))
(algorithms.ts:231-276).
"""
from __future__ import annotations

import ctypes as C
import weakref
from typing import Sequence, Tuple

import numpy as np

from ._lib import RangeError, check, default_ctx, ket_batch_template, ket_op, ket_param_binding, lib


def batch_qaoa(instances: Sequence[Tuple[int, Sequence[Tuple[int, int]], Sequence[float], Sequence[float]]],
               use_graph: bool = True, tune: bool = False) -> np.ndarray:
    """Expected cut <C> of every instance (n, edges, gamma, beta).  tune: pick
    the launch shape with the autotuner (ket_b200/autotune.py), timing the
    candidates on this batch the first time a batch of its shape is seen."""
    if not instances:
        return np.zeros(0)
    if tune:
        from . import autotune
        cfg = autotune.cached_batch_config(instances) or autotune.tune_batch_qaoa(instances)
        autotune.set_batch_config(cfg["block_threads"], cfg["tile_bits"])
    return _run(instances, use_graph)


def _run(instances, use_graph: bool) -> np.ndarray:
    p = len(instances[0][2])
    ns, nes, eoff, edges, gam, bet = [], [], [], [], [], []
    for n, e, g, b in instances:
        if len(g) != p or len(b) != p:
            raise TypeError("every instance needs the same number of gamma and beta angles")
        ns.append(n)
        nes.append(len(e))
        eoff.append(len(edges) // 2)
        for u, v in e:
            edges += [u, v]
        gam += list(g)
        bet += list(b)
    N = len(instances)
    n_a = np.ascontiguousarray(ns, dtype=np.int32)
    ne_a = np.ascontiguousarray(nes, dtype=np.int32)
    eo_a = np.ascontiguousarray(eoff, dtype=np.int64)
    ed_a = np.ascontiguousarray(edges or [0, 0], dtype=np.int32)
    g_a = np.ascontiguousarray(gam or [0.0], dtype=np.float64)
    b_a = np.ascontiguousarray(bet or [0.0], dtype=np.float64)
    out = np.zeros(N)
    ip = lambda a: a.ctypes.data_as(C.POINTER(C.c_int))
    dp = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    check(lib().ket_batch_qaoa(default_ctx(), N, ip(n_a), ip(ne_a), eo_a.ctypes.data_as(C.POINTER(C.c_int64)),
                               ip(ed_a), p, dp(g_a), dp(b_a), 1 if use_graph else 0, dp(out)))
    return out


def batch_vqe(templates, instances, use_graph: bool = True) -> np.ndarray:
    """vqe() energies of many parameterised circuits in one launch.

    templates: [(ansatz, hamiltonian)], an ansatz being a function params ->
    Circuit (AnsatzFn or any callable) on at most 13 qubits and a hamiltonian
    a PauliTerm list, as vqe(ansatz(params), hamiltonian) takes them
    (algorithms.ts:301-336).  instances: [(template index, params)].  Returns
    energy[i] = vqe(ansatz_t(params_i), H_t) for every instance, computed with
    the reference's per-gate pruning; instances of different templates may
    differ in width, gates and Hamiltonian.  Each ansatz is traced once and
    kept while the ansatz object lives, so it must build the same gate list
    on every call (as the adjoint's trace requires)."""
    from .adjoint import _terms
    if not instances:
        return np.zeros(0)
    which = [t for t, _ in instances]
    params = [v for _, v in instances]
    if not (0 <= min(which) and max(which) < len(templates)):
        bad = next(t for t in which if not 0 <= t < len(templates))
        raise RangeError(f"instance template index {bad} out of range")
    it = np.ascontiguousarray(which, dtype=np.int32)
    lens = list(map(len, params))
    nparams = max(lens)
    first = dict(zip(reversed(which), reversed(params)))  # (the first instance of a template stays)
    tmpl = (ket_batch_template * max(1, len(templates)))()
    all_ops, all_mats, all_binds, coeffs, pauli = [], [], [], [], []
    nops = nmats = nbinds = npauli = 0
    for j, (ansatz, ham) in enumerate(templates):
        p0 = first.get(j)
        if p0 is None:
            p0 = [0.3] * getattr(ansatz, "paramCount", nparams)
        n, ops, mats, binds = _traced(ansatz, p0)
        terms = _terms(ham, n)
        tmpl[j].nqubits, tmpl[j].nops, tmpl[j].nbinds, tmpl[j].nterms = n, len(ops), len(binds), len(terms)
        tmpl[j].op_first, tmpl[j].bind_first = nops, nbinds
        tmpl[j].term_first, tmpl[j].pauli_first = len(coeffs), npauli
        if nmats:
            ops = ops.copy()
            ops["mat"][ops["mat"] >= 0] += nmats
        all_ops.append(ops.view(np.uint8))  # (plain bytes join faster than structures)
        all_mats.append(mats)
        all_binds.append(binds.view(np.uint8))
        nops, nmats, nbinds = nops + len(ops), nmats + len(mats), nbinds + len(binds)
        for c, o in terms:
            coeffs.append(c)
            pauli.append(o)
            npauli += len(o)
    join = lambda a: a[0] if len(a) == 1 else np.concatenate(a)
    ops_a = join(all_ops) if nops else np.zeros(1, dtype=_OP)
    binds_a = join(all_binds) if nbinds else np.zeros(1, dtype=_BIND)
    mats = np.concatenate(all_mats + [np.zeros(1, dtype=np.complex128)]).view(np.float64)
    cf = np.ascontiguousarray(coeffs or [0.0], dtype=np.float64)
    ps = "".join(pauli).encode()
    th = _theta(params, lens, nparams)
    out = np.zeros(len(instances))
    dp = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    check(lib().ket_batch_vqe(default_ctx(), len(templates), tmpl, ops_a.ctypes.data_as(C.POINTER(ket_op)), dp(mats),
                              mats.size // 2, binds_a.ctypes.data_as(C.POINTER(ket_param_binding)), dp(cf), ps,
                              len(instances), it.ctypes.data_as(C.POINTER(C.c_int)), dp(th), max(nparams, 1),
                              1 if use_graph else 0, dp(out)))
    return out


def _theta(params, lens, nparams):
    """Every instance's parameters at the start of its row of max(nparams, 1)."""
    n = len(params)
    if nparams and min(lens) == nparams:
        return np.ascontiguousarray(np.asarray(params, dtype=np.float64).reshape(-1))
    th = np.zeros((n, max(nparams, 1)))
    if n > 64 and isinstance(params[0], np.ndarray):  # (arrays join faster than a loop copies them; lists do not)
        try:
            flat = np.concatenate(params)
        except ValueError:  # (of shapes that do not join)
            flat = None
        # plain numbers only: what else an assignment converts or refuses is left to it
        if flat is not None and flat.ndim == 1 and flat.dtype.kind in "biuf":
            th[np.arange(th.shape[1]) < np.asarray(lens)[:, None]] = flat
            return th
    for row, v in zip(th, params):
        row[:len(v)] = v
    return th


# Traced templates, kept per ansatz function while it lives: a parameter sweep
# calls batch_vqe again and again with the same ansatze, and tracing (two
# builds of the circuit) costs more host time than the batch's kernel.  They are
# kept as arrays of the ABI's structures, so that a call joins them with a few
# array operations.
_TRACE_CACHE = weakref.WeakKeyDictionary()
_OP = np.dtype(ket_op)
_BIND = np.dtype(ket_param_binding)


def _traced(ansatz, p0):
    """(n, ket_op array, matrices, bindings) of an ansatz, traced once."""
    from .adjoint import trace
    from .circuit import ops_to_abi
    key = len(p0)
    try:
        hit = _TRACE_CACHE.get(ansatz, {}).get(key)
    except TypeError:  # not weak-referenceable: trace every time
        hit = None
    if hit is None:
        n, ops, binds = trace(ansatz, [float(v) for v in p0])
        arr, m, k = ops_to_abi(ops)
        b = np.zeros(len(binds), dtype=_BIND)
        for i, v in enumerate(binds):
            b[i]["op"], b[i]["gate"], b[i]["param"], b[i]["scale"], b[i]["shift"] = v
        hit = (n, np.frombuffer(arr, dtype=_OP, count=k).copy(), m, b)
        try:
            _TRACE_CACHE.setdefault(ansatz, {})[key] = hit
        except TypeError:
            pass
    return hit
