"""A GMRES cycle whose start vector arrives in separate columns while the cycle
runs, against the in-place call (one array, sent the same way) and the cycle
from zero: a cycle of one step (all of it sent after the steps), one longer
than a batch of steps, one that ends early, and start vectors in other orders
and strides.  Start plus increment is one rounded sum per value, so all agree
exactly."""
import ctypes as C

import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import api
from oversetdevfort_b200 import mesh as M

pytestmark = pytest.mark.gpu


def _in_place(ctx, system, tol, kspace, start):
    s = np.array(start, order="F")
    info = F.OvsGmresInfo()
    F.check(ctx.lib.ovs_gmres(ctx.h, system, tol, kspace, 1, s.ctypes.data_as(C.POINTER(C.c_double)), C.byref(info)),
            "ovs_gmres")
    return s, info


@pytest.mark.parametrize("tol,kspace", [(1e-30, 1), (1e-30, 21), (1e-3, 60)])
@pytest.mark.parametrize("dims", [(1, 1, 2), (9, 7, 12)])
def test_start_columns(dims, tol, kspace):
    ctx = api.Context.from_case(M.quench_case(M.box_tet(*dims), "start", seed=3))
    N = ctx.N
    rng = np.random.default_rng(5)
    kspace = min(kspace, N // 2)
    for kernel, system, nf in ((F.OVS_ASM_NSVOF, F.OVS_SYS_NSVOF, 5), (F.OVS_ASM_TEM, F.OVS_SYS_TEM, 1)):
        ctx.assemble(kernel, 6, F.OVS_FP64)
        start = np.asfortranarray(rng.standard_normal((N, nf)))
        keep = start.copy()
        ref, ir = _in_place(ctx, system, tol, kspace, start)
        inc, _ = ctx.gmres(system, tol, kspace, 1, np.zeros((N, nf)))
        if not ctx.get_rhs(system).any():   # (the smallest mesh's temperature) the solution is set to zero
            assert nf == 1 and not ref.any() and not inc.any()
            continue
        np.testing.assert_allclose(ref, start + inc, rtol=0, atol=1e-14 * max(1.0, np.abs(ref).max()))
        for form in (start, np.ascontiguousarray(start), np.repeat(start, 2, axis=0)[::2]):
            s, info = ctx.gmres(system, tol, kspace, 1, form)
            assert info.iterations == ir.iterations and np.array_equal(s, ref)
        if nf == 5:
            u, p, ls, _ = api.SparseGMRES_ns_conv(ctx, tol, kspace, 1, start[:, :3], start[:, 3], start[:, 4:])
            assert np.array_equal(np.column_stack([u, p, ls]), ref)
        else:
            t, _ = api.SparseGMRES_tem(ctx, tol, kspace, 1, start[:, 0])
            assert np.array_equal(t, ref[:, 0])
        assert np.array_equal(start, keep)
    with pytest.raises(ValueError):
        api.SparseGMRES_tem(ctx, tol, kspace, 1, np.zeros(N + 1))
    ctx.close()
