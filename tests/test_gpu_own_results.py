"""The SparseGMRES_* calls return arrays of their own: one that is kept does not
keep the others, (N, 3) results are column-major, and a later call does not
change them.  Columns of one array and columns apart get the same values."""
import ctypes as C

import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import api
from oversetdevfort_b200 import mesh as M

pytestmark = pytest.mark.gpu


def test_results_own_their_memory():
    ctx = api.Context.from_case(M.quench_case(M.box_tet(4, 3, 3), "own", seed=3))
    N = ctx.N
    ctx.assemble(F.OVS_ASM_NSVOF, 6, F.OVS_FP64)
    ctx.assemble(F.OVS_ASM_TEM, 6, F.OVS_FP64)
    ctx.assemble(F.OVS_ASM_NS, 6, F.OVS_FP64)
    rng = np.random.default_rng(5)
    u0, p0, f0, t0 = (rng.standard_normal(s) for s in ((N, 3), N, N, N))
    runs = {"ns": lambda: api.SparseGMRES_up(ctx, 1e-3, 20, 1, u0, p0)[:-1],
            "nsvof": lambda: api.SparseGMRES_ns_conv(ctx, 1e-3, 20, 1, u0, p0, f0)[:-1],
            "tem": lambda: api.SparseGMRES_tem(ctx, 1e-3, 20, 1, t0)[:-1]}
    for kind, run in runs.items():
        out = run()
        keep = [x.copy() for x in out]
        again = run()
        for x, k, y in zip(out, keep, again):
            assert x.flags.owndata and x.flags.f_contiguous and x.flags.writeable, kind
            np.testing.assert_array_equal(x, k)
            np.testing.assert_array_equal(x, y)
            y[...] = 0.0
            np.testing.assert_array_equal(x, k)
    ctx.close()


def test_one_array_and_columns_apart_agree():
    ctx = api.Context.from_case(M.quench_case(M.box_tet(4, 3, 3), "own", seed=3))
    ctx.assemble(F.OVS_ASM_NSVOF, 6, F.OVS_FP64)
    start = np.random.default_rng(6).standard_normal((5, ctx.N))
    dp = C.POINTER(C.c_double)
    cols = (dp * 5)(*(r.ctypes.data_as(dp) for r in start))
    one, info = np.empty((5, ctx.N)), F.OvsGmresInfo()
    F.check(ctx.lib.ovs_gmres_from(ctx.h, F.OVS_SYS_NSVOF, 1e-3, 20, 1, cols, one.ctypes.data_as(dp), C.byref(info)),
            "ovs_gmres_from")
    apart = np.full((10, ctx.N), 7.0)   # every second row, so that no two columns follow one another
    out = (dp * 5)(*(r.ctypes.data_as(dp) for r in apart[::2]))
    F.check(ctx.lib.ovs_gmres_columns(ctx.h, F.OVS_SYS_NSVOF, 1e-3, 20, 1, cols, out, C.byref(info)),
            "ovs_gmres_columns")
    np.testing.assert_array_equal(apart[::2], one)
    assert (apart[1::2] == 7.0).all()
    out[4] = None
    assert ctx.lib.ovs_gmres_columns(ctx.h, F.OVS_SYS_NSVOF, 1e-3, 20, 1, cols, out, C.byref(info)) == F.OVS_ERR_ARG
    assert ctx.lib.ovs_gmres_columns(ctx.h, F.OVS_SYS_NSVOF, 1e-3, 401, 1, cols, cols, C.byref(info)) == F.OVS_ERR_ARG
    ctx.close()
