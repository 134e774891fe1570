"""The reverse-mode VJP of the residual with every option of the element
routines on: phase change, discontinuity capturing in all three fields,
solid elements, Dirichlet nodes, mesh motion, VOF values outside [0, 1], and
element counts that leave a block of 128 threads and a group of 16 nodes
partly filled.  Central differences along seeded directions (h = 1e-6 of each
field's scale): truncation is O(h^2) and the rounding of the contracted
residuals about 1e-16 / h of their magnitude, so 1e-5 relative to the sum of
the directional terms' magnitudes."""
import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import mesh as M
from oversetdevfort_b200.adjoint import residuals
from oversetdevfort_b200.api import Context

pytestmark = pytest.mark.gpu

COLS = {"xg": slice(0, 3), "ug": slice(3, 6), "pg": 6, "phig": 7, "tg": 8, "acg": slice(9, 12), "rphig": 12,
        "rtg": 13}


def _low_word(n):
    """1 with n in the low half of its bits (what e3DC_beta2 reads as an integer)."""
    return float(np.array([0x3FF0000000000000 + n], dtype=np.uint64).view(np.float64)[0])


@pytest.mark.parametrize("dims,seed,kdc", [((1, 1, 1), 5, False), ((3, 2, 2), 6, False), ((4, 3, 3), 7, False),
                                           ((4, 3, 3), 8, True)])
def test_vjp_with_every_option(dims, seed, kdc):
    case = M.random_case(*dims, seed=seed, solid_frac=0.2)
    rng = np.random.default_rng(100 + seed)
    if kdc:
        # the property blend of NS_kdc is exact only where the VOF value is
        # clamped, so all of it is gas here
        case.params.update(ns_kdc_w=_low_word(40), ns_kdc_a=_low_word(70))
        for n in ("phig", "phigold"):
            case.state[n][:] = rng.uniform(1.1, 1.6, case.mesh.nnode)
    ctx = Context.from_case(case)
    st0 = {n: ctx.get_field(n).copy() for n in COLS}
    scale = {n: 0.02 * min(1.0 / dims[0], 0.8 / dims[1]) if n == "xg" else max(np.abs(a).max(), 1e-3)
             for n, a in st0.items()}
    v1, v2 = rng.standard_normal((ctx.N, 5)), rng.standard_normal(ctx.N)
    for kernel, cot in ((F.OVS_ASM_NSVOF, v1), (F.OVS_ASM_TEM, v2)):
        g = ctx.residual_vjp(kernel, cot)
        for n, a in st0.items():
            w = scale[n] * rng.standard_normal(a.shape)
            vals = []
            for sgn in (1.0, -1.0):
                ctx.set_field(n, a + sgn * 1e-6 * w)
                r = residuals(ctx)[0 if kernel == F.OVS_ASM_NSVOF else 1]
                vals.append(np.sum(cot * r))
            ctx.set_field(n, a)
            terms = g[:, COLS[n]] * w
            fd = (vals[0] - vals[1]) / 2e-6
            assert abs(fd - terms.sum()) <= 1e-5 * np.abs(terms).sum() + 1e-9 * abs(vals[0]), (n, fd, terms.sum())
    ctx.close()
