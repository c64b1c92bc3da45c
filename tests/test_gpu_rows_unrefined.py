"""Few-right-hand-side sweeps (rows.cu) with columns assembled once per node, one sweep
per solve: refinement would shrink an error of the sweeps themselves.  Counts of
right-hand sides that give every chunk width of these kernels, carriers (two per
instance) and Poisson."""
import pytest

import oracle
import pecs_gb300 as pg
from helpers import to_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,degree,pairing,n_inst", [(40, 2, 0, 3), (44, 2, 1, 4), (24, 2, 0, 5), (24, 2, 1, 6),
                                                     (31, 1, 0, 8), (31, 1, 1, 12), (24, 2, 0, 13)])
def test_single_sweeps_solve(pecs_lib, n, degree, pairing, n_inst):
    """Relative residuals.  The same factors applied on the host in one sweep leave 1.5e-12
    in FP64 and 7e-4 in FP32 at most on meshes of 31 to 60 cells (random and smooth
    right-hand sides, both matrices): 1e-10 and 1e-2 with room.  A lost update or a
    wrong column leaves about one."""
    base = oracle.half_cell_params(n_refine=3, degree=degree, poisson_pairing=pairing)
    base.nx_semi, base.nx_elec, base.ny = n, n - 3, n - 1
    Ps = [to_lib(base.copy(phi_app=0.1 * i)) for i in range(n_inst)]
    for prec, tol in ((pg.PREC_FP64, 1e-10), (pg.PREC_FP32_IR, 1e-2)):
        ctx = pg.Context(Ps, precision=prec, ir_max_iters=-1, flow_sweep=-1)
        ctx.initialize()
        ctx.step(1)
        for which in (0, 1):
            assert ctx.solve_residual(which) < tol, (prec, which)
