"""batch_vqe()'s parameters and template indices on their way to the engine: what is
converted and what is refused does not depend on the number of instances or on the
container they come in."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

import ket_b200 as K
from ket_b200 import batch as B


@pytest.fixture
def sent(monkeypatch):
    """The parameter rows and template indices handed to ket_batch_vqe."""
    got = {}

    class Lib:
        @staticmethod
        def ket_batch_vqe(ctx, ntmpl, tmpl, ops, mats, nmat, binds, cf, ps, ninst, which, th, nparams, graph, out):
            got["theta"] = np.ctypeslib.as_array(th, (ninst, nparams)).copy()
            got["which"] = np.ctypeslib.as_array(which, (ninst,)).copy()
            return 0

    monkeypatch.setattr(B, "lib", lambda: Lib)
    monkeypatch.setattr(B, "default_ctx", lambda: None)
    return got


def templates():
    one = lambda p: K.Circuit(2).rx(p[0], 0).ry(p[1], 1)
    two = lambda p: K.Circuit(3).rx(p[0], 0).ry(p[1], 1).rz(p[2], 2)
    return [(one, [(1.0, "ZZ")]), (two, [(1.0, "ZZX")])]


FORMS = {
    "list": list,
    "tuple": tuple,
    "array": np.asarray,
    "float32": lambda v: np.asarray(v, dtype=np.float32),
    "ints": lambda v: [int(8 * x) for x in v],
    "fractions": lambda v: [Fraction(x) for x in v],
    "texts": lambda v: [str(x) for x in v],
}


@pytest.mark.parametrize("count", [2, 64, 65, 130])
@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("ragged", [False, True])
def test_rows(sent, count, form, ragged):
    r = np.random.default_rng(count)
    which = [i % 2 if ragged else 0 for i in range(count)]
    values = [np.round(r.uniform(-3, 3, 2 + t) * 64) / 64 for t in which]
    inst = [(t, FORMS[form](v.tolist())) for t, v in zip(which, values)]
    B.batch_vqe(templates() if ragged else templates()[:1], inst)
    want = np.zeros((count, 3 if ragged else 2))
    for row, v in zip(want, values):
        row[:len(v)] = (8 * v).astype(int) if form == "ints" else v
    assert np.array_equal(sent["theta"], want) and sent["which"].tolist() == which


@pytest.mark.parametrize("count", [2, 64, 65])
def test_columns_of_equal_length(sent, count):
    """A column of parameters, one entry a row."""
    v = np.random.default_rng(1).uniform(-3, 3, (count, 2))
    T = templates()[:1]
    B.batch_vqe(T, [(0, [0.1, 0.2])] * count)  # traced by plain numbers
    B.batch_vqe(T, [(0, x.reshape(2, 1)) for x in v])
    assert np.array_equal(sent["theta"], v)


@pytest.mark.parametrize("count", [3, 64, 65, 130])
@pytest.mark.parametrize("ragged", [False, True])
def test_complex_parameters_are_refused(sent, count, ragged):
    T = templates()
    B.batch_vqe(T, [(0, [0.1, 0.2]), (1, [0.1, 0.2, 0.3])])  # traced by plain numbers
    inst = [(i % 2, [0.1, 0.2, 0.3][:2 + i % 2]) if ragged else (0, [0.1, 0.2]) for i in range(count - 1)]
    with pytest.raises(TypeError):
        B.batch_vqe(T if ragged else T[:1], inst + [(0, [0.1, 0.2 + 0.5j])])


@pytest.mark.parametrize("count", [3, 70])
@pytest.mark.parametrize("bad", [-1, 2, 1 << 40])
def test_index_out_of_range(sent, count, bad):
    inst = [(0, [0.1, 0.2])] * (count - 1) + [(bad, [0.1, 0.2])]
    with pytest.raises(K.RangeError):
        B.batch_vqe(templates(), inst)


@pytest.mark.parametrize("count", [3, 70])
def test_instances_are_pairs(sent, count):
    with pytest.raises(ValueError):
        B.batch_vqe(templates()[:1], [(0, [0.1, 0.2])] * count + [(0, [0.1, 0.2], "more")])
