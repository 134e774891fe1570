"""Cycles of large Krylov spaces, where the orthogonalization changes shape with
the step: rows of T longer than two lanes' worth (65), fewer than eight threads
per column of T in the step's finish (130), one (400, the largest space), more
shared memory than the 48 KB every kernel may take (200), and a workspace that
grows and serves smaller cycles after.  Against the one-launch variant (plain
modified Gram-Schmidt).

Tolerance.  The two variants lose orthogonality alike, and the solution of a
cycle that has not converged is the least-squares one over the same space: the
iterates agree to the rounding of k steps times the condition of the space.  A
diagonally dominant system set by hand (off-diagonal row sums at most half the
diagonal, condition of P^-1 A at most 3) is solved with a tolerance of zero; the
residual reaches rounding after about 50 steps and every iterate after that is
the solution to rounding: 1e-12 of its largest entry in FP64 (k eps cond =
400 * 1.1e-16 * 3 = 1.3e-13, times 8 for both sides' sums), and in FP32, whose
basis and products round at 6e-8, 400 * 6e-8 * 3 = 7e-5."""
import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import mesh as M
from oversetdevfort_b200.api import Context

pytestmark = pytest.mark.gpu


def _system(ctx, seed):
    """A temperature system with off-diagonal row sums of half the diagonal, and its dense solution."""
    col, row = ctx.get_pattern()
    ptr, idx = col.astype(np.int64) - 1, row.astype(np.int64) - 1
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(ctx.N), np.diff(ptr))
    vals = rng.uniform(-1.0, 1.0, len(idx))
    off = rows != idx
    sums = np.bincount(rows[off], np.abs(vals[off]), ctx.N)
    vals = np.where(off, 0.5 * vals / sums[rows], 1.0)
    vals32 = vals.astype(np.float32).astype(np.float64)
    rhs = rng.standard_normal(ctx.N).astype(np.float32).astype(np.float64)
    A = np.zeros((ctx.N, ctx.N))
    A[rows, idx] = vals32
    for prec in (F.OVS_FP64, F.OVS_FP32):
        ctx.set_lhs(F.OVS_SYS_TEM, prec, F.OVS_BLK_TEM, vals32)
        ctx.set_rhs(F.OVS_SYS_TEM, prec, rhs)
    return np.linalg.solve(A, rhs)


def _both(ctx, kspace, kmin):
    zero = np.zeros((ctx.N, 1))
    out = []
    for fused in (0, 1):
        ctx.set_option(F.OVS_OPT_ARNOLDI_FUSED, fused)
        s, info = ctx.gmres(F.OVS_SYS_TEM, 1e-30, kspace, kmin, zero)
        out.append((s[:, 0], info.iterations))
    ctx.set_option(F.OVS_OPT_ARNOLDI_FUSED, 0)
    return out


def test_large_spaces_against_the_one_launch_variant_and_the_dense_solution():
    ctx = Context.from_case(M.quench_case(M.box_tet(12, 9, 8), "large", seed=3))   # 1,170 nodes
    want = _system(ctx, 7)
    scale = np.abs(want).max()
    first = None
    for kspace in (65, 130, 200, 400, 12, 400):
        (a, na), (b, nb) = _both(ctx, kspace, kspace)
        assert na == nb == kspace
        assert np.abs(a - b).max() <= 1e-12 * scale
        if kspace >= 130:
            assert np.abs(a - want).max() <= 1e-12 * scale
        if kspace == 400:   # the second time, after a small cycle: the same bits
            first = a if first is None else first
            np.testing.assert_array_equal(a, first)
        x, info = ctx.solve(F.OVS_SYS_TEM, F.OVS_FP32, 1e-30, kspace=kspace, max_cycles=1)
        assert info.cycles == 1
        if kspace >= 65:
            assert np.abs(x[:, 0] - want).max() <= 7e-5 * scale
    ctx.close()
