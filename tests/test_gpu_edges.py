"""The edge pass of the tet assembly where its geometry changes: fewer rows
than a tile (16), one tile, one row more, two tiles and one row more, several, with the nodes and
elements renumbered at random (the pass follows the coordinates, not the
numbers), nodes that no element holds, and rows of very unequal degree; all
kernels, both precisions, against the oracle.  Tolerances as the parity tests:
1e-12 in FP64, 1e-5 in FP32, of the largest entry of each block.  A second
assembly gives the same bits, and so does a context whose pattern is built
twice."""
import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import mesh as M
from oversetdevfort_b200.api import Context

pytestmark = pytest.mark.gpu

KERNELS = {"nsvof": (F.OVS_ASM_NSVOF, F.OVS_SYS_NSVOF), "tem": (F.OVS_ASM_TEM, F.OVS_SYS_TEM),
           "ns": (F.OVS_ASM_NS, F.OVS_SYS_NS)}


def _renumber(case, rng, extra):
    """The case with random node and element numbers and `extra` nodes without elements."""
    m, N = case.mesh, case.mesh.nnode
    new = rng.permutation(N + extra)[:N]
    x = np.zeros((N + extra, 3), order="F")
    x[:] = rng.uniform(0.0, 1.0, x.shape)
    x[new] = m.xg
    perm = rng.permutation(m.nelem)
    ien = np.asfortranarray((new[m.ien.astype(np.int64) - 1] + 1).astype(np.int32)[perm])
    st = {}
    for k, v in case.state.items():
        st[k] = np.zeros((N + extra,) + v.shape[1:], order="F")
        st[k][new] = v
    ibc = np.zeros((N + extra, 8), dtype=np.int32, order="F")
    ibc[new] = case.ibc
    mesh = M.Mesh(x, ien, np.ascontiguousarray(m.elm_id[perm]), [np.zeros(0, np.int64)] * 6, m.dims, m.lengths)
    return M.Case(case.name, mesh, case.params, st, ibc, case.kernel)


@pytest.mark.parametrize("kind", list(KERNELS))
@pytest.mark.parametrize("dims,extra", [((1, 1, 1), 0), ((1, 1, 3), 0), ((1, 1, 3), 1), ((3, 1, 3), 0), ((10, 2, 0), 0), ((4, 3, 3), 3), ((9, 7, 6), 5)])
def test_edge_pass_against_the_oracle(oracle, kind, dims, extra):
    kernel, system = KERNELS[kind]
    if dims[2] == 0:
        dims = (10, 2, 1)                      # 66 nodes: two tiles and two rows
    rng = np.random.default_rng(sum(dims) + extra)
    case = _renumber(M.random_case(*dims, seed=31, kernel=kernel), rng, extra)
    oc = oracle.OracleCase(case)
    if kind == "ns":
        oc.assemble_navsto(6)
    else:
        oc.assemble_quenching(6, 7)
    ref = oc.system(kind)
    ctx = Context.from_case(case)
    for prec, tol in ((F.OVS_FP64, 1e-12), (F.OVS_FP32, 1e-5)):
        ctx.assemble(kernel, 6, prec)
        got = ctx.get_system(system, prec)
        for k, v in got.items():
            want = np.asarray(ref[k]).reshape(v.shape)
            assert np.abs(v - want).max() <= tol * max(np.abs(want).max(), 1e-300), (k, prec)
        ctx.build_pattern()
        ctx.assemble(kernel, 6, prec)
        again = ctx.get_system(system, prec)
        for k in got:
            np.testing.assert_array_equal(got[k], again[k], err_msg=k)
    ctx.close()
