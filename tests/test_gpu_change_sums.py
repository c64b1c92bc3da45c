"""The element-wise kernels of the batched increment solves (engine.cu): the changes of
a step that its scatters add up for the steady-state test, and the residual with four
right-hand sides per lane, at sizes with partial tiles of dofs, partial tiles of
columns and rows with fewer entries than are fetched at a time."""
import numpy as np
import pytest

import oracle
import pecs_gb300 as pg
from helpers import rel_err, to_lib
from test_gpu_parity import _panel_instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nxe,ny,degree,n_inst", [(5, 7, 3, 1, 33), (8, 8, 8, 1, 48), (5, 3, 7, 2, 50),
                                                     (16, 12, 17, 1, 64)])
def test_march_reports_the_change_of_its_last_step(pecs_lib, nx, nxe, ny, degree, n_inst):
    """rel against |u5 - u4| / |u5| of the states.  Squares are of values truncated to 24
    bits (2 * 2^-23 each), a thread adds four of them in FP32 (3 * 2^-24), the rest is
    FP64: 2e-7 in the ratio of the roots, 1e-6 with room.  The march and plain steps
    launch the same solves: the same states bit for bit.  The refined solves' states
    (the other residual kernels) are within 2e-6: 1e-6 of FP64 each, what the mixed mode keeps."""
    base = oracle.half_cell_params(n_refine=3, degree=degree)
    base.nx_semi, base.nx_elec, base.ny = nx, nxe, ny
    Ps = [to_lib(P) for P in _panel_instances(n_inst, base)]
    mk = lambda inc: pg.Context(Ps, precision=pg.PREC_FP32_MIXED, increment_solves=inc, autotune=False)
    a, b, c = mk(True), mk(True), mk(False)
    for ctx in (a, b, c):
        ctx.initialize()
    steps, rel = a.run_to_steady_state(5, 1e-30, 50)
    assert np.all(np.asarray(steps) == 5)
    b.step(4)
    old = {f: [b.get_state(f, i) for i in range(n_inst)] for f in b.fields()}
    b.step(1)
    c.step(5)
    for i in range(n_inst):
        want = 0.0
        for f in b.fields():
            u = b.get_state(f, i)
            assert np.array_equal(u, a.get_state(f, i)), (f, i)
            assert rel_err(c.get_state(f, i), u) < 2e-6, (f, i)
            want = max(want, np.linalg.norm(u - old[f][i]) / np.linalg.norm(u))
        assert abs(rel[i] - want) < 1e-6 * want, (i, rel[i], want)
