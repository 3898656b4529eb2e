"""States of two contexts, each with a stream of its own: a copy from one into the
other follows what was queued on the source, from its allocation on."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Context:
    def __init__(self):
        from ket_b200 import _lib
        self.L, self.h = _lib, C.c_void_p()
        _lib.check(_lib.lib().ket_ctx_create(0, C.byref(self.h)))
        self.states = []

    def state(self, n, precision=0):
        h = C.c_void_p()
        self.L.check(self.L.lib().ket_state_alloc(self.h, n, precision, C.byref(h)))
        self.states.append(h)
        return h

    def close(self):
        for s in self.states:
            self.L.check(self.L.lib().ket_state_free(s))
        self.L.check(self.L.lib().ket_ctx_destroy(self.h))


@pytest.mark.parametrize("n", [1, 12, 27])
@pytest.mark.parametrize("precision", [0, 1])
def test_copy_follows_the_source(n, precision):
    from ket_b200 import _lib
    L = _lib.lib()
    a, b = Context(), Context()
    try:
        src, dst = a.state(n, precision), b.state(n, precision)
        _lib.check(L.ket_state_copy(dst, src))  # straight after the allocation
        last = (1 << n) - 1
        idx = (C.c_uint64 * 2)(0, last)
        out = np.zeros(4)
        norm = C.c_double()
        for k in range(6):
            want = last if k % 2 == 0 else 0
            _lib.check(L.ket_state_set_basis(src, want))
            _lib.check(L.ket_state_copy(dst, src))
            _lib.check(L.ket_amplitudes(dst, idx, 2, out.ctypes.data_as(C.POINTER(C.c_double))))
            _lib.check(L.ket_norm2(dst, C.byref(norm)))
            assert out.tolist() == ([0, 0, 1, 0] if want else [1, 0, 0, 0]) and norm.value == 1.0
    finally:
        b.close()
        a.close()
