"""The hexahedral element and row passes where their geometry changes: one
element, rows of up to 8 elements in chunks of 4, nodes without elements, a
fan of hexahedra around one edge (rows of 12 elements and 50 columns: three
chunks, sums carried between them), random numbering, solid elements, Dirichlet
nodes and phase change, against the oracle: 1e-12 in FP64, 1e-5 in FP32, of
the largest entry of each block, and the same bits on a second run."""
import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import mesh as M
from oversetdevfort_b200.api import Context

pytestmark = pytest.mark.gpu

KERNELS = {"nsvof": (F.OVS_ASM_NSVOF, F.OVS_SYS_NSVOF), "tem": (F.OVS_ASM_TEM, F.OVS_SYS_TEM)}


def _with_mesh(case, xg, ien, rng):
    N, E = xg.shape[0], ien.shape[0]
    st = {k: np.asfortranarray(rng.uniform(v.min(), v.max(), (N,) + v.shape[1:])) for k, v in case.state.items()}
    h = np.abs(xg[ien[:, 0] - 1] - xg[ien[:, 6] - 1]).min() + 0.1
    for k in ("dg", "dgold"):
        st[k][:] = rng.uniform(-0.02, 0.02, st[k].shape) * h
    elm = np.where(rng.random(E) < 0.2, 101, 102).astype(np.int32)
    ibc = np.asfortranarray((rng.random((N, 8)) < 0.2).astype(np.int32))
    mesh = M.Mesh(np.asfortranarray(xg), np.asfortranarray(ien.astype(np.int32)), elm, [np.zeros(0, np.int64)] * 6,
                  (E, 1, 1), (1.0, 1.0, 1.0))
    return M.Case(case.name, mesh, case.params, st, ibc, case.kernel)


def _fan(n, rng):
    """n hexahedra around the z axis: quadrilaterals (axis, rim 2j, 2j+1, 2j+2) over two planes."""
    k = np.arange(2 * n)
    ang = 2 * np.pi * k / (2 * n)
    rim = np.stack([np.cos(ang), np.sin(ang)], axis=1) * np.where(k % 2, 1.3, 1.0)[:, None]
    xy = np.concatenate([np.zeros((1, 2)), rim])
    x = np.concatenate([np.concatenate([xy, np.full((len(xy), 1), z)], axis=1) for z in (0.0, 1.0)])
    m = len(xy)
    ien = np.zeros((n, 8), dtype=np.int64)
    for j in range(n):
        q = [0, 1 + 2 * j, 1 + (2 * j + 1) % (2 * n), 1 + (2 * j + 2) % (2 * n)]   # counter-clockwise
        corner = {(0, 0): q[0], (1, 0): q[1], (1, 1): q[2], (0, 1): q[3]}
        for a, (i, jj, kk) in enumerate(M._HEX):
            ien[j, a] = corner[(i, jj)] + m * kk
    return x, ien + 1


@pytest.mark.parametrize("kind", list(KERNELS))
@pytest.mark.parametrize("shape", ["one", "box", "renumbered", "fan5", "fan12"])
def test_hex_passes_against_the_oracle(oracle, kind, shape):
    kernel, system = KERNELS[kind]
    rng = np.random.default_rng(17)
    case = M.random_case(*{"one": (1, 1, 1), "box": (5, 3, 4)}.get(shape, (3, 4, 3)), seed=12, kernel=F.OVS_ASM_NSVOF,
                         hex=True)
    if shape == "renumbered":
        m = case.mesh
        new = rng.permutation(m.nnode + 4)[:m.nnode]
        x = rng.uniform(0.0, 1.0, (m.nnode + 4, 3))
        x[new] = m.xg
        case = _with_mesh(case, x, (new[m.ien.astype(np.int64) - 1] + 1)[rng.permutation(m.nelem)], rng)
    elif shape.startswith("fan"):
        case = _with_mesh(case, *_fan(int(shape[3:]), rng), rng)
    oc = oracle.OracleCase(case)
    oc.assemble_quenching(6, 7)
    ref = oc.system(kind)
    ctx = Context.from_case(case)
    if shape == "fan12":
        assert np.diff(ctx.get_pattern()[0]).max() == 50
    for prec, tol in ((F.OVS_FP64, 1e-12), (F.OVS_FP32, 1e-5)):
        ctx.assemble(kernel, 6, prec)
        got = ctx.get_system(system, prec)
        for k, v in got.items():
            want = np.asarray(ref[k]).reshape(v.shape)
            assert np.abs(v - want).max() <= tol * max(np.abs(want).max(), 1e-300), (k, prec)
        ctx.assemble(kernel, 6, prec)
        again = ctx.get_system(system, prec)
        for k in got:
            np.testing.assert_array_equal(got[k], again[k], err_msg=k)
    ctx.close()
