"""Vector-only assembly (the residual evaluation of the Newton loop) takes its
own element and row passes: the same right-hand side as the matrix-and-vector
pass (which the parity tests pin to the oracle) and, in FP64, as the oracle, for every kernel, element type and precision, at sizes
below and across a block of rows (32 nodes) and of elements (128, hexahedra
64), with solid elements, Dirichlet nodes and phase change; and the matrix
assembled before stays as it was.  Tolerances as the full pass's: 1e-12 in
FP64, 1e-5 in FP32, of the largest entry of each field."""
import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import mesh as M
from oversetdevfort_b200.api import Context, calculate_residual

pytestmark = pytest.mark.gpu


def _close(a, b, tol):
    for f in range(b.shape[1]):
        assert np.abs(a[:, f] - b[:, f]).max() <= tol * max(np.abs(b[:, f]).max(), 1e-300)


@pytest.mark.parametrize("prec,tol", [(F.OVS_FP64, 1e-12), (F.OVS_FP32, 1e-5)])
@pytest.mark.parametrize("hexa,dims", [(False, (1, 1, 1)), (False, (4, 3, 3)), (False, (7, 5, 6)),
                                       (True, (1, 1, 1)), (True, (4, 3, 3)), (True, (6, 5, 4))])
def test_vector_only_matches_the_full_pass(oracle, hexa, dims, prec, tol):
    kernels = [(F.OVS_ASM_NSVOF, F.OVS_SYS_NSVOF, "nsvof"), (F.OVS_ASM_TEM, F.OVS_SYS_TEM, "tem")]
    if not hexa:
        kernels.append((F.OVS_ASM_NS, F.OVS_SYS_NS, "ns"))
    for kernel, system, kind in kernels:
        case = M.random_case(*dims, seed=11, kernel=kernel, hex=hexa)
        oc = oracle.OracleCase(case)
        if kind == "ns":
            oc.assemble_navsto(6)
        else:
            oc.assemble_quenching(6, 7)
        ref = oc.system(kind)["rhs"].reshape(case.mesh.nnode, -1)
        with Context.from_case(case) as ctx:
            ctx.assemble(kernel, F.OVS_TENSOR_MAT | F.OVS_TENSOR_VEC, prec)
            full, block = ctx.get_rhs(system, prec), F.OVS_BLK_TEM if kind == "tem" else F.OVS_BLK_K11
            mat = ctx.get_lhs(system, prec, block)
            ctx.assemble(kernel, F.OVS_TENSOR_VEC, prec)
            rhs = ctx.get_rhs(system, prec)
            np.testing.assert_array_equal(ctx.get_lhs(system, prec, block), mat)
            norms = calculate_residual(ctx, prec)
        _close(rhs, full, tol)
        if prec == F.OVS_FP64:
            _close(rhs, ref, tol)
        sq = (rhs ** 2).sum(axis=0)
        want = [0.0, 0.0, 0.0, sq[0]] if kind == "tem" else [sq[:3].sum(), sq[3], sq[4] if kind == "nsvof" else 0.0, 0.0]
        np.testing.assert_allclose(norms, want, rtol=1e-12)
