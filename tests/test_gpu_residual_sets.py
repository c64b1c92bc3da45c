"""Refinement residuals in FP32 pairs (engine.cu) of banks whose sets have different
widths: electrons and holes of one region with distinct mobilities are sets of n columns
each, the other region's one set of 2 n.  Each set takes the kernel of its own width."""
import pytest

import oracle
import pecs_gb300 as pg
from helpers import rel_err, to_lib
from test_gpu_parity import _panel_instances

pytestmark = pytest.mark.gpu


def _contexts(n_inst, mu, **kw):
    base = oracle.half_cell_params(n_refine=3)
    base.mu = mu
    Ps = [to_lib(P) for P in _panel_instances(n_inst, base)]
    return Ps, pg.Context(Ps, precision=pg.PREC_FP32_MIXED, autotune=False, flow_sweep=-1, **kw)


@pytest.mark.parametrize("increment", [False, True])
@pytest.mark.parametrize("mu", [(1.0, 0.5, 1.0, 1.0), (1.0, 1.0, 2.0, 0.7)])
def test_each_set_takes_the_kernel_of_its_width(pecs_lib, mu, increment):
    """48 instances: sets of 48, 48 and 96, the last with four right-hand sides per lane and
    the others in a launch of their own; 47 (94) and 96 (96 and 192): one launch.  The
    states are within 1e-6 of FP64's, what the mixed mode keeps."""
    launches = {n: _contexts(n, mu, increment_solves=increment)[1].info().launches_per_step for n in (47, 48, 96)}
    assert launches[48] == launches[47] + 1 == launches[96] + 1, launches
    Ps, ctx = _contexts(48, mu, increment_solves=increment)
    ctx.initialize()
    ctx.step(4)
    for i in (0, 23, 47):
        one = pg.Context(Ps[i])
        one.initialize()
        one.step(4)
        for f in ctx.fields():
            assert rel_err(ctx.get_state(f, i), one.get_state(f)) < 1e-6, (i, f)
