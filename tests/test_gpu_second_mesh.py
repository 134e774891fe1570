"""A context that takes a second mesh of as many nodes and elements: a refused
one leaves no mesh to assemble on (its connectivity has replaced the earlier
one by then), whatever was built before."""
import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import mesh as M
from oversetdevfort_b200.api import Context

pytestmark = pytest.mark.gpu


def _remeshed(m, ien):
    return M.Mesh(m.xg, np.asfortranarray(ien.astype(np.int32)), m.elm_id, m.faces, m.dims, m.lengths)


def test_a_refused_mesh_leaves_none():
    case = M.random_case(3, 3, 2, seed=8, kernel=F.OVS_ASM_NSVOF)
    ctx = Context.from_case(case)
    ctx.assemble(F.OVS_ASM_NSVOF, 6, F.OVS_FP64)
    ref = ctx.get_system(F.OVS_SYS_NSVOF)
    bad = case.mesh.ien.copy()
    bad[5, 2] = bad[5, 0]   # an element that repeats a node
    with pytest.raises(F.OvsError) as e:
        ctx.upload_mesh(_remeshed(case.mesh, bad))
    assert e.value.status == F.OVS_ERR_ARG
    for call in (ctx.build_pattern, lambda: ctx.assemble(F.OVS_ASM_NSVOF, 6, F.OVS_FP64),
                 lambda: ctx.residual_vjp(F.OVS_ASM_NSVOF, np.ones((ctx.N, 5)))):
        with pytest.raises(F.OvsError) as e:
            call()
        assert e.value.status == F.OVS_ERR_STATE
    ctx.upload_mesh(case.mesh)
    ctx.build_pattern()
    ctx.assemble(F.OVS_ASM_NSVOF, 6, F.OVS_FP64)
    got = ctx.get_system(F.OVS_SYS_NSVOF)
    for k in ref:
        np.testing.assert_array_equal(got[k], ref[k], err_msg=k)
    ctx.close()
