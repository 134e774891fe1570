"""Two host threads, each with a context of its own on one device, where calls
of one need more dynamic shared memory than calls of the other: that limit
belongs to the kernel, not to the context, so a call must not lower it under
another thread's launches.  Krylov spaces of 200 and 3 (a 200-step cycle asks
for 60.8 KB in its last steps), and hexahedral row passes of rows of 27 and of
8 columns.  Every call runs to its end and gives the bits it gives alone.
The systems are small: all blocks of both threads fit the device at once."""
import threading

import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import mesh as M
from oversetdevfort_b200.api import Context

pytestmark = pytest.mark.gpu


def _beside(work, other):
    """work() here while another thread repeats other()."""
    stop, failed = threading.Event(), []

    def loop():
        try:
            while not stop.is_set():
                other()
        except Exception as e:   # reported by the caller's thread
            failed.append(e)

    t = threading.Thread(target=loop)
    t.start()
    try:
        work()
    finally:
        stop.set()
        t.join()
    assert not failed, failed


def test_krylov_spaces_of_two_threads():
    a = Context.from_case(M.quench_case(M.box_tet(5, 4, 3), "large_space", seed=3))
    b = Context.from_case(M.quench_case(M.box_tet(4, 3, 3), "small_space", seed=4))
    zero = [np.zeros((c.N, 5)) for c in (a, b)]
    for c in (a, b):
        c.assemble(F.OVS_ASM_NSVOF, 6, F.OVS_FP64)
    ref_a, info = a.gmres(F.OVS_SYS_NSVOF, 1e-30, 200, 200, zero[0])
    ref_b, _ = b.gmres(F.OVS_SYS_NSVOF, 1e-30, 3, 1, zero[1])
    assert info.iterations == 200

    def large():
        for _ in range(30):
            s, i = a.gmres(F.OVS_SYS_NSVOF, 1e-30, 200, 200, zero[0])
            assert i.iterations == 200
            np.testing.assert_array_equal(s, ref_a)

    def small():
        np.testing.assert_array_equal(b.gmres(F.OVS_SYS_NSVOF, 1e-30, 3, 1, zero[1])[0], ref_b)

    _beside(large, small)
    a.close()
    b.close()


@pytest.mark.parametrize("kernel,system", [(F.OVS_ASM_NSVOF, F.OVS_SYS_NSVOF), (F.OVS_ASM_TEM, F.OVS_SYS_TEM)])
def test_hexahedral_rows_of_two_threads(kernel, system):
    a = Context.from_case(M.random_case(3, 3, 3, seed=5, kernel=kernel, hex=True))
    b = Context.from_case(M.random_case(1, 1, 1, seed=6, kernel=kernel, hex=True))
    refs = []
    for c in (a, b):
        c.assemble(kernel, 6, F.OVS_FP64)
        refs.append(c.get_system(system))

    def large():
        for _ in range(1000):
            a.assemble(kernel, 6, F.OVS_FP64)

    _beside(large, lambda: b.assemble(kernel, 6, F.OVS_FP64))
    for c, ref in zip((a, b), refs):
        got = c.get_system(system)
        for k in ref:
            np.testing.assert_array_equal(got[k], ref[k], err_msg=k)
        c.close()
