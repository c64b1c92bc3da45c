"""pecs_set_instances: many short vectors are uploaded together."""
import time

import pytest

import oracle
import pecs_gb300 as pg
from helpers import to_lib
from test_gpu_parity import _panel_instances

pytestmark = pytest.mark.gpu


def _params(n_inst, refine, seed):
    base = oracle.half_cell_params(n_refine=refine)
    return [to_lib(P.copy(phi_app=0.001 * (i + seed))) for i, P in enumerate(_panel_instances(n_inst, base))]


@pytest.mark.parametrize("n_inst,refine", [(1, 2), (300, 3), (20, 5), (3, 6)])
def test_vectors_arrive_as_in_a_new_context(pecs_lib, n_inst, refine):
    """Short, long and single vectors, more of them than one piece holds: the states after a
    step are those of a context created with the parameters, bit for bit."""
    a = pg.Context(_params(n_inst, refine, 0), autotune=False, flow_sweep=-1)
    b = pg.Context(_params(n_inst, refine, 7), autotune=False, flow_sweep=-1)
    a.set_instances(_params(n_inst, refine, 7))
    for ctx in (a, b):
        ctx.initialize()
        ctx.step(1)
    for i in range(n_inst):
        for f in a.fields():
            assert (a.get_state(f, i) == b.get_state(f, i)).all(), (i, f)


def test_many_small_instances_cost_what_their_cells_do(pecs_lib):
    """256 instances of 8x8 cells against 16 of 32x32: as many cells and bytes.  A copy for
    each of their 2,800 vectors made it ten times as long; four times is allowed."""
    best = {}
    for n_inst, refine in ((256, 3), (16, 5)):
        P = _params(n_inst, refine, 0)
        ctx = pg.Context(P, autotune=False, flow_sweep=-1)
        arr = (pg._ffi.pecs_params * n_inst)(*[p.to_c() for p in P])
        best[n_inst] = 1e9
        for _ in range(8):
            t = time.perf_counter()
            pg._ffi.check(pg.lib().pecs_set_instances(ctx._h, arr, n_inst))
            best[n_inst] = min(best[n_inst], time.perf_counter() - t)
    assert best[256] < 4 * best[16], best
