"""Few-right-hand-side sweeps (rows.cu) of levels with large fronts: tiles staged through
two buffers, and columns assembled for three and four right-hand sides.  Relative
residuals of the solves: FP64 factors with one refinement 1e-10 (the large-mesh tests'),
FP32 factors refined with FP64 residuals the same."""
import pytest

import oracle
import pecs_gb300 as pg
from helpers import to_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,degree,pairing,n_inst", [(40, 2, 0, 3), (40, 2, 0, 4), (44, 2, 1, 1), (44, 2, 1, 2),
                                                     (60, 2, 1, 3)])
def test_large_fronts_solve(pecs_lib, n, degree, pairing, n_inst):
    base = oracle.half_cell_params(n_refine=3, degree=degree, poisson_pairing=pairing)
    base.nx_semi, base.nx_elec, base.ny = n, n - 3, n - 1
    Ps = [to_lib(base.copy(phi_app=0.1 * i)) for i in range(n_inst)]
    for prec, iters in ((pg.PREC_FP64, 0), (pg.PREC_FP32_IR, 3)):
        ctx = pg.Context(Ps, precision=prec, ir_max_iters=iters, flow_sweep=-1)
        ctx.initialize()
        ctx.step(2)
        for which in (0, 1):
            assert ctx.solve_residual(which) < 1e-10, (prec, which)
