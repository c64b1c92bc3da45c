"""Device memory of contexts whose banks take the many-right-hand-side kernels (solve.cu):
one form of the factors stays once the kernels are chosen, and factor_bytes counts it."""
import numpy as np
import pytest

import oracle
import pecs_gb300 as pg
from helpers import to_lib
from test_gpu_parity import _panel_instances

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def _held(torch, n_inst, refine, **kw):
    """Device bytes of a context, factor values left out."""
    Ps = [to_lib(P) for P in _panel_instances(n_inst, oracle.half_cell_params(n_refine=refine))]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ctx = pg.Context(Ps, **kw)
    used = free - torch.cuda.mem_get_info()[0]
    return used - ctx.info().factor_bytes, ctx.info().factor_bytes, ctx


@pytest.mark.parametrize("kw", [{"flow_sweep": -1}, {"flow_sweep": -1, "autotune": False}, {"autotune": False}, {}])
def test_one_form_of_the_factors_stays(pecs_lib, kw):
    """16 instances (32 right-hand sides per carrier factor, the panel kernels) against 15
    (30, the others): a context's memory without its factors grows with the instances
    alone, one fifteenth.  48 MiB are allowed for the plans' index lists and the
    allocations' granularity; a second form of these carrier factors takes more."""
    torch = pytest.importorskip("torch")
    for n_inst in (15, 16):  # kernels and workspaces that are loaded once
        _held(torch, n_inst, 3, **kw)
    few, f_few, a = _held(torch, 15, 6, **kw)
    many, f_many, b = _held(torch, 16, 6, **kw)
    if list(b.info().flow_rpl) != [0, 0]:
        pytest.skip("a flow sweep was chosen: it keeps a form of its own")
    print(few / MIB, f_few / MIB, many / MIB, f_many / MIB)
    assert f_many > 2 * 48 * MIB and 0.8 < f_many / f_few < 1.2  # a second form could not hide in the allowance
    assert many < few * 16 / 15 + 48 * MIB
    for ctx in (a, b):
        ctx.initialize()
        ctx.step(1)
        assert ctx.solve_residual(0) < 1e-10
