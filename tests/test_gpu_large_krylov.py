"""Cycles of large Krylov spaces, where the orthogonalization changes shape with
the step: rows of T longer than two lanes' worth (65), fewer than eight threads
per column of T in the step's finish (130), one (400, the largest space), more
shared memory than the 48 KB every kernel may take (200), and a workspace that
grows and serves smaller cycles after.  Against the one-launch variant (plain
modified Gram-Schmidt), the dense solution and dense iterates.

Tolerance of the converged cycles.  The two variants lose orthogonality alike, and the solution of a
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


def _snake(nx, ny, nz):
    """The nodes of a box mesh, each one a neighbour of the one before."""
    path = []
    for k in range(nz + 1):
        for j in range(ny + 1) if k % 2 == 0 else range(ny, -1, -1):
            line = [(i, j, k) for i in range(nx + 1)]
            path += line if len(path) % (2 * (nx + 1)) == 0 else line[::-1]
    return path


def _iterate(A, b, k):
    """The k-th GMRES iterate from zero: least squares over an Arnoldi basis orthogonalized twice, FP64."""
    V = np.zeros((len(b), k + 1))
    H = np.zeros((k + 1, k))
    V[:, 0] = b / np.linalg.norm(b)
    for j in range(k):
        w = A @ V[:, j]
        for _ in range(2):
            h = V[:, :j + 1].T @ w
            H[:j + 1, j] += h
            w -= V[:, :j + 1] @ h
        H[j + 1, j] = np.linalg.norm(w)
        V[:, j + 1] = w / H[j + 1, j]
    e = np.zeros(k + 1)
    e[0] = np.linalg.norm(b)
    return V[:, :k] @ np.linalg.lstsq(H, e, rcond=None)[0]


def test_large_spaces_without_convergence():
    """A = I + 0.98 S, S the shift along a path of neighbouring nodes: the
    residual falls by 0.98 a step, so that no cycle up to 400 steps ends early
    in either precision (0.98^400 = 3e-4, FP32 stops at 1e-6).  Its condition is
    at most 1.98 / 0.02 = 99: the iterates agree to k eps cond, 400 * 6e-8 * 99 =
    2.4e-3 of the largest entry in FP32, 400 * 1.1e-16 * 99 = 4.4e-12 in FP64,
    times 8 there as above."""
    dims = (12, 9, 8)
    case = M.quench_case(M.box_tet(*dims), "shift", seed=3)
    ctx = Context.from_case(case)
    N = ctx.N
    xyz = np.rint(case.mesh.xg * np.array(dims)).astype(int)
    node = {tuple(p): i for i, p in enumerate(xyz)}
    path = np.array([node[p] for p in _snake(*dims)])
    assert len(set(path.tolist())) == N
    a = float(np.float32(0.98))
    A = np.eye(N)
    A[path[1:], path[:-1]] = a
    col, row = ctx.get_pattern()
    ptr, idx = col.astype(np.int64) - 1, row.astype(np.int64) - 1
    vals = A[np.repeat(np.arange(N), np.diff(ptr)), idx]
    assert np.count_nonzero(vals) == 2 * N - 1   # the pattern holds every step of the path
    rhs = np.random.default_rng(9).standard_normal(N).astype(np.float32).astype(np.float64)
    for prec in (F.OVS_FP64, F.OVS_FP32):
        ctx.set_lhs(F.OVS_SYS_TEM, prec, F.OVS_BLK_TEM, vals)
        ctx.set_rhs(F.OVS_SYS_TEM, prec, rhs)
    for kspace in (65, 130, 200, 400):
        want = _iterate(A, rhs, kspace)
        scale = np.abs(want).max()
        for fused in (0, 1):
            ctx.set_option(F.OVS_OPT_ARNOLDI_FUSED, fused)
            x, info = ctx.gmres(F.OVS_SYS_TEM, 1e-30, kspace, 1, np.zeros((N, 1)))
            assert info.iterations == kspace
            assert np.abs(x[:, 0] - want).max() <= 8 * 4.4e-12 * scale, (kspace, fused)
            x, info = ctx.solve(F.OVS_SYS_TEM, F.OVS_FP32, 1e-30, kspace=kspace, max_cycles=1)
            assert info.iterations == kspace
            assert np.abs(x[:, 0] - want).max() <= 2.4e-3 * scale, (kspace, fused)
    ctx.close()
