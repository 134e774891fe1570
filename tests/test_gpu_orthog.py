"""The orthogonalization kernel of the Arnoldi iterations against the
one-launch variant (OVS_OPT_ARNOLDI_FUSED, plain modified Gram-Schmidt, which
the oracle tests pin) and the oracle's cycle, where its geometry changes: one
vector, a group of eight less and more one, more vectors than a block has
warps, vectors shorter than a sub-chunk, a ragged last sub-chunk, the switch
from one to four values per lane (303,104 values on 148 SMs), and the
temperature system's scalar rows.  Both variants solve the same system in
FP64 and differ by rounding: 1e-9 of the largest entry, as for the full-size
case."""
import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import mesh as M
from oversetdevfort_b200.api import Context

pytestmark = pytest.mark.gpu

TOL = 1e-9


def _cycle(ctx, system, kspace, fused):
    ctx.set_option(F.OVS_OPT_ARNOLDI_FUSED, fused)
    nf = 1 if system == F.OVS_SYS_TEM else 5
    return ctx.gmres(system, 1e-30, kspace, 1, np.zeros((ctx.N, nf)))


@pytest.mark.parametrize("kspace", [1, 2, 7, 8, 9, 17, 33])
@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 4, 3), (11, 9, 13)])
def test_orthog_matches_the_fused_variant_and_the_oracle(oracle, dims, kspace):
    case = M.quench_case(M.box_tet(*dims), "orthog", seed=3)
    rng = np.random.default_rng(7)
    case.state["ug"][:] = rng.uniform(-0.01, 0.01, case.state["ug"].shape)
    case.state["rtg"][:] = rng.uniform(-10.0, 10.0, case.mesh.nnode)
    ctx = Context.from_case(case)
    oc = oracle.OracleCase(case)
    oc.assemble_quenching(6, 7)
    for kernel, system, kind in ((F.OVS_ASM_NSVOF, F.OVS_SYS_NSVOF, "nsvof"), (F.OVS_ASM_TEM, F.OVS_SYS_TEM, "tem")):
        ctx.assemble(kernel, 6, F.OVS_FP64)
        # a space no larger than the system, so that no cycle breaks down
        n = ctx.N * (1 if kind == "tem" else 2)
        k = min(kspace, n // 2)
        a, ia = _cycle(ctx, system, k, 0)
        b, ib = _cycle(ctx, system, k, 1)
        ref, it, _, _ = oc.gmres(kind, 1e-30, k, 1)
        assert ia.iterations == ib.iterations == it == k
        np.testing.assert_allclose(ia.res0, ib.res0, rtol=1e-12)
        scale = np.abs(ref).max()
        assert np.abs(a - b).max() <= TOL * scale
        assert np.abs(a.reshape(ref.shape) - ref).max() <= TOL * scale
    ctx.close()


@pytest.mark.parametrize("dims", [(38, 38, 38), (39, 39, 38), (40, 39, 39)])
def test_orthog_at_the_switch_of_values_per_lane(dims):
    ctx = Context.from_case(M.quench_case(M.box_tet(*dims), "orthog_switch", seed=3))
    ctx.assemble(F.OVS_ASM_NSVOF, 6, F.OVS_FP64)
    a, ia = _cycle(ctx, F.OVS_SYS_NSVOF, 20, 0)
    b, ib = _cycle(ctx, F.OVS_SYS_NSVOF, 20, 1)
    assert ia.iterations == ib.iterations == 20
    assert np.abs(a - b).max() <= TOL * np.abs(b).max()
    # FP32 basis: one cycle of the FP32-assembled system, as the full-size case
    ctx.assemble(F.OVS_ASM_NSVOF, 6, F.OVS_FP32)
    out = []
    for fused in (0, 1):
        ctx.set_option(F.OVS_OPT_ARNOLDI_FUSED, fused)
        out.append(ctx.solve(F.OVS_SYS_NSVOF, F.OVS_FP32, 1e-30, kspace=20, max_cycles=1)[0])
    assert np.abs(out[0] - out[1]).max() <= 1e-4 * np.abs(out[1]).max()
    ctx.close()


@pytest.mark.parametrize("dims", [(77, 78, 77), (78, 78, 77)])
def test_orthog_at_the_switch_to_eight_values_per_lane(dims):
    """FP32: 2,424,832 values on 148 SMs, ragged lengths on both sides.  Four
    steps: the variants then differ by a few roundings of the basis vectors
    (6e-8 each) times the condition of a 4x4 Hessenberg matrix, below 1e-5 of
    the largest entry; over 20 steps the one-launch variant's own error against
    FP64 reaches 9e-5 at this size."""
    ctx = Context.from_case(M.quench_case(M.box_tet(*dims), "orthog_switch8", seed=3))
    ctx.assemble(F.OVS_ASM_NSVOF, 6, F.OVS_FP32)
    out = []
    for fused in (0, 1):
        ctx.set_option(F.OVS_OPT_ARNOLDI_FUSED, fused)
        out.append(ctx.solve(F.OVS_SYS_NSVOF, F.OVS_FP32, 1e-30, kspace=4, max_cycles=1)[0])
    assert np.abs(out[1]).max() > 0.0
    assert np.abs(out[0] - out[1]).max() <= 1e-5 * np.abs(out[1]).max()
    ctx.close()


@pytest.mark.parametrize("n,kspace", [(1, 4), (2, 9), (4, 12)])
def test_ns_rows_by_nodes_match_the_oracle(oracle, n, kspace):
    """The (u,p) system's product with vectors by nodes: 8, 27 and 125 rows, one
    warp of eight rows, a ragged last one, several blocks of 64 threads.  The
    enclosed cavity leaves the pressure's constant to rounding: compared without."""
    case = M.config1(n)
    ctx = Context.from_case(case)
    oc = oracle.OracleCase(case)
    oc.assemble_navsto(6)
    ctx.assemble(F.OVS_ASM_NS, 6, F.OVS_FP64)
    ref, it, _, _ = oc.gmres("ns", 1e-12, kspace, 1)
    s, info = ctx.gmres(F.OVS_SYS_NS, 1e-12, kspace, 1, np.zeros((ctx.N, 4)))
    assert info.iterations == it
    d = s - ref
    d[:, 3] -= d[:, 3].mean()
    assert np.abs(d).max() <= TOL * np.abs(ref).max()
    ctx.close()
