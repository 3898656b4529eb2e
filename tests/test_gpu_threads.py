"""Threads with a context each, more of them than cores: every call's answer is that of a
thread alone."""
import ctypes as C
import os
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Worker(threading.Thread):
    def __init__(self, n, abi, calls):
        from ket_b200 import _lib
        super().__init__()
        self.L, self.lib, self.n, self.abi, self.calls = _lib, _lib.lib(), n, abi, calls
        self.error, self.out = None, []
        self.ctx, self.st = C.c_void_p(), C.c_void_p()
        _lib.check(self.lib.ket_ctx_create(0, C.byref(self.ctx)))
        _lib.check(self.lib.ket_state_alloc(self.ctx, n, 0, C.byref(self.st)))

    def run(self):
        try:
            arr, m, k = self.abi
            mv = np.ascontiguousarray(m).view(np.float64)
            o = self.L.exec_opts()
            for _ in range(self.calls):
                self.L.check(self.lib.ket_state_set_basis(self.st, 0))
                self.L.check(self.lib.ket_apply_ops(self.st, arr, k, mv.ctypes.data_as(C.POINTER(C.c_double)), m.size,
                                                    C.byref(o)))
                a = np.empty(1 << self.n, dtype=np.complex128)
                self.L.check(self.lib.ket_state_get_amplitudes(self.st, 0, 1 << self.n,
                                                               a.view(np.float64).ctypes.data_as(C.POINTER(C.c_double))))
                self.out.append(a)
        except Exception as e:  # (told to the test's own thread)
            self.error = e

    def close(self):
        self.L.check(self.lib.ket_state_free(self.st))
        self.L.check(self.lib.ket_ctx_destroy(self.ctx))


@pytest.mark.parametrize("cores", [1, 2])
@pytest.mark.parametrize("n,calls", [(6, 40), (16, 10), (20, 4)])
def test_threads_share_cores(n, calls, cores):
    from ket_b200 import workloads as W
    abi = [W.brickwork_circuit(n, 5, s)[0].to_abi() for s in range(4)]
    alone = [Worker(n, a, 1) for a in abi]
    for w in alone:
        w.run()
    ours = os.sched_getaffinity(0)
    os.sched_setaffinity(0, set(sorted(ours)[:cores]))
    crowd = [Worker(n, a, calls) for a in abi]
    try:
        for w in crowd:
            w.start()
        for w in crowd:
            w.join()
        for w, one in zip(crowd, alone):
            assert w.error is None and one.error is None and len(w.out) == calls
            assert all(np.array_equal(a, one.out[0]) for a in w.out)
    finally:
        os.sched_setaffinity(0, ours)
        for w in crowd + alone:
            w.close()
