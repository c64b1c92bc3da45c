"""Level sweeps of banks with many right-hand sides (solve.cu, k_panel_tiles) where
their tiles, chunks of columns and groups of right-hand sides have edges: counts of
right-hand sides that are odd, even or multiples of four, just past a group of 32, 64 or
128, and columns staged a few at a time.  Against the same instances one by one (the
few-right-hand-side kernels)."""
import pytest

import oracle
import pecs_gb300 as pg
from helpers import rel_err, to_lib
from test_gpu_parity import _panel_instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [1, 2])
@pytest.mark.parametrize("n_inst,chunk,min_ctas", [(16, 0, 0), (17, 1, 0), (33, 0, 0), (33, 7, 1), (66, 16, 0), (67, 0, 1)])
def test_level_sweeps_match_single_instances(pecs_lib, n_inst, chunk, min_ctas, degree):
    """FP64: both paths round at 1e-16 times the factors' growth, 1e-11 over two steps
    with room.  FP32 factors with refinement: 1e-6, what the mixed mode keeps."""
    Ps = [to_lib(P) for P in _panel_instances(n_inst, oracle.half_cell_params(n_refine=3, degree=degree))]
    for prec, tol in ((pg.PREC_FP64, 1e-11), (pg.PREC_FP32_MIXED, 1e-6)):
        for autotune in (False, True):
            ctx = pg.Context(Ps, precision=prec, flow_sweep=-1, autotune=autotune, panel_chunk=chunk,
                             panel_min_ctas=min_ctas)
            ctx.initialize()
            ctx.step(2)
            for i in (0, n_inst // 2, n_inst - 1):
                one = pg.Context(Ps[i])
                one.initialize()
                one.step(2)
                for f in ctx.fields():
                    assert rel_err(ctx.get_state(f, i), one.get_state(f)) < tol, (prec, autotune, i, f)
