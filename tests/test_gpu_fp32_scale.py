"""The scale of an FP32 Krylov vector is applied unrounded: the new vector is
w / |v_k| in the length that the coefficients were formed with, not in that of
a reciprocal rounded to FP32.  A temperature system is set by hand so that
every value of the two-step cycle is a small whole number but the reciprocal
1/14: with e a node, q four of its neighbours in two neighbouring pairs and f a
node next to them all,
  A e = e + 7 sum q,   A q = q - (q's partner) + 7 f + e,   b = e,
the slots are e, 7 sum q (length 14), and A (7 sum q) / 14 = 2 e + 14 f; the
solution of the two-step cycle is 196/39396 e + 196/39396 sum q.  In FP32,
196 * fl(1/14) is not 14 (it is 6.8e-8 off), 196 * (1/14) rounded once is.
What remains is a few dozen FP64 roundings: 1e-13 of the largest entry.
Sizes: one value per lane, and four (303,104 values on 148 SMs)."""
import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import mesh as M
from oversetdevfort_b200.api import Context

pytestmark = pytest.mark.gpu


def _nodes(ptr, idx):
    """e, f and two neighbouring pairs next to both, all neighbours of one another as the matrix needs."""
    near = lambda i: set(idx[ptr[i]:ptr[i + 1]].tolist()) - {i}
    for e in range(len(ptr) - 1):
        for f in sorted(near(e)):
            pairs, used = [], set()
            both = sorted(near(e) & near(f))
            for p in both:
                for q in both:
                    if p < q and not {p, q} & used and q in near(p):
                        pairs.append((p, q))
                        used |= {p, q}
            if len(pairs) >= 2:
                return e, f, pairs[:2]
    raise AssertionError("no such nodes")


@pytest.mark.parametrize("dims", [(5, 4, 3), (68, 68, 67)])
def test_the_scale_of_an_fp32_vector_is_not_rounded(dims):
    assert np.float32(196) * np.float32(1 / 14) != 14 and np.float32(196 * (1 / 14)) == 14
    ctx = Context.from_case(M.quench_case(M.box_tet(*dims), "scale", seed=3))
    col, row = ctx.get_pattern()
    ptr, idx = col.astype(np.int64) - 1, row.astype(np.int64) - 1
    e, f, pairs = _nodes(ptr, idx)
    vals = np.zeros(len(idx))
    vals[np.flatnonzero(idx == np.repeat(np.arange(ctx.N), np.diff(ptr)))] = 1.0

    def put(i, j, v):
        k = ptr[i] + np.searchsorted(idx[ptr[i]:ptr[i + 1]], j)
        assert idx[k] == j
        vals[k] = v

    for p, q in pairs:
        for a, b in ((p, q), (q, p)):
            put(a, e, 7.0)
            put(b, a, -1.0)
            put(f, a, 7.0)
            put(e, a, 1.0)
    rhs = np.zeros(ctx.N)
    rhs[e] = 1.0
    ctx.set_lhs(F.OVS_SYS_TEM, F.OVS_FP32, F.OVS_BLK_TEM, vals)
    ctx.set_rhs(F.OVS_SYS_TEM, F.OVS_FP32, rhs)
    x, info = ctx.solve(F.OVS_SYS_TEM, F.OVS_FP32, 1e-30, kspace=2, max_cycles=1)
    assert info.iterations == 2
    want = np.zeros(ctx.N)
    want[[e, *pairs[0], *pairs[1]]] = 196.0 / 39396.0
    assert np.abs(x[:, 0] - want).max() <= 1e-13 * want.max()
    ctx.close()
