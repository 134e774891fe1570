"""A context that takes a second mesh of as many nodes and elements: a refused
one leaves no mesh to assemble on (its connectivity has replaced the earlier
one by then), whatever was built before; a pattern of another length drops the
matrices that the earlier one sized, the same pattern again keeps them, and a
refused build leaves none."""
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


def _shuffled(case, seed):
    """The case on a mesh of as many nodes and elements, of nodes drawn at random (a longer pattern)."""
    m, rng = case.mesh, np.random.default_rng(seed)
    x = np.asfortranarray(rng.uniform(0.0, 1.0, m.xg.shape))
    ien = np.array([rng.permutation(m.nnode)[:4] + 1 for _ in range(m.nelem)])
    for e in ien:   # positive volume
        a, b, c, d = x[e - 1]
        if np.dot(a - d, np.cross(b - d, c - d)) < 0.0:
            e[:2] = e[1::-1].copy()
    mesh = M.Mesh(x, np.asfortranarray(ien.astype(np.int32)), m.elm_id, m.faces, m.dims, m.lengths)
    return M.Case(case.name, mesh, case.params, case.state, case.ibc, case.kernel)


def _all(ctx, prec):
    out = {}
    for kernel, system in ((F.OVS_ASM_NSVOF, F.OVS_SYS_NSVOF), (F.OVS_ASM_TEM, F.OVS_SYS_TEM), (F.OVS_ASM_NS, F.OVS_SYS_NS)):
        ctx.assemble(kernel, 6, prec)
        out.update({(system, k): v for k, v in ctx.get_system(system, prec).items()})
    if prec == F.OVS_FP64:
        out["t"] = ctx.gmres_transposed(F.OVS_SYS_TEM, np.arange(ctx.N) + 1.0, 1e-8, 20)[0]
    return out


def _take(ctx, case):
    ctx.upload_mesh(case.mesh)
    ctx.build_pattern()


def test_a_longer_pattern_after_a_shorter_one_and_back():
    """Short, long, short, long again: each as a context of its own gives it,
    whether or not something was assembled in between; a solve before the new
    matrix exists is an error of call order."""
    short = M.random_case(4, 3, 3, seed=9, kernel=F.OVS_ASM_NSVOF)   # 80 nodes
    long = _shuffled(short, 10)
    want = {}
    for name, case in (("short", short), ("long", long)):
        with Context.from_case(case) as c:
            want[name] = (c.icnt, {p: _all(c, p) for p in (F.OVS_FP64, F.OVS_FP32)})
    assert want["long"][0] > want["short"][0]
    ctx = Context.from_case(short)
    cases = {"short": short, "long": long}
    for name, used in (("short", True), ("long", True), ("short", True), ("long", False), ("short", True), ("long", True)):
        _take(ctx, cases[name])
        assert ctx.icnt == want[name][0]
        for system in (F.OVS_SYS_NSVOF, F.OVS_SYS_TEM):
            with pytest.raises(F.OvsError) as e:
                ctx.gmres(system, 1e-3, 5, 1, np.zeros((ctx.N, 5 if system == F.OVS_SYS_NSVOF else 1)))
            assert e.value.status == F.OVS_ERR_STATE
        if not used:
            continue
        for prec in (F.OVS_FP64, F.OVS_FP32):
            got = _all(ctx, prec)
            for k, v in want[name][1][prec].items():
                np.testing.assert_array_equal(got[k], v, err_msg=str(k))
    ctx.close()


def test_the_same_pattern_again_keeps_the_matrix_and_a_refused_one_does_not():
    case = M.random_case(4, 3, 3, seed=9, kernel=F.OVS_ASM_NSVOF)
    ctx = Context.from_case(case)
    ctx.assemble(F.OVS_ASM_NSVOF, 6, F.OVS_FP64)
    x = np.random.default_rng(1).standard_normal((ctx.N, 5))
    y = ctx.spmv(F.OVS_SYS_NSVOF, F.OVS_FP64, x)
    _take(ctx, case)
    np.testing.assert_array_equal(ctx.spmv(F.OVS_SYS_NSVOF, F.OVS_FP64, x), y)
    bad = case.mesh.ien.copy()
    bad[3, 1] = ctx.N + 1   # no such node
    ctx.upload_mesh(_remeshed(case.mesh, bad))
    with pytest.raises(F.OvsError) as e:
        ctx.build_pattern()
    assert e.value.status == F.OVS_ERR_ARG
    with pytest.raises(F.OvsError) as e:
        ctx.spmv(F.OVS_SYS_NSVOF, F.OVS_FP64, x)
    assert e.value.status == F.OVS_ERR_STATE
    ctx.close()
