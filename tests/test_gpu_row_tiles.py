"""The edge pass at two tiles of 16 rows and one row more (33) and at two tiles
and two rows (34), against the oracle as the other tile edges; and the former
row-pass options, which are accepted in their old ranges and change nothing
(the pass they are set for is the one that the oracle pins here).  Tolerances as
the parity tests: 1e-12 in FP64, 1e-5 in FP32, of the largest entry of each
block."""
import numpy as np
import pytest

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import mesh as M
from oversetdevfort_b200.api import Context
from test_gpu_edges import KERNELS, _renumber

pytestmark = pytest.mark.gpu

OPTIONS = {F.OVS_OPT_ROWS_STAGED: (0, 1, 7), F.OVS_OPT_ROWS_GATHER: (0, 1, -1), F.OVS_OPT_ROWS_TILED: (1, 0, 3),
           F.OVS_OPT_TILE_ELEMS: (4, 96, 4000)}


@pytest.mark.parametrize("kind", list(KERNELS))
@pytest.mark.parametrize("extra", [1, 2])
def test_two_tiles_and_a_little_more(oracle, kind, extra):
    kernel, system = KERNELS[kind]
    case = _renumber(M.random_case(3, 1, 3, seed=37, kernel=kernel), np.random.default_rng(extra), extra)
    assert case.mesh.nnode == 32 + extra
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
        for option, values in OPTIONS.items():
            for value in values:
                ctx.set_option(option, value)
                ctx.assemble(kernel, 6, prec)
                for k, v in ctx.get_system(system, prec).items():
                    np.testing.assert_array_equal(v, got[k], err_msg=f"{option} {value} {k}")
    for value in (3, 4001):
        with pytest.raises(F.OvsError) as e:
            ctx.set_option(F.OVS_OPT_TILE_ELEMS, value)
        assert e.value.status == F.OVS_ERR_ARG
    ctx.close()
