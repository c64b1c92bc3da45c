"""Network predictions written over their inputs (nn.cu): y_dev at x_dev, and a few rows
off it either way.  The outputs must be the same bits as into memory of their own."""
import pytest

from pecs_gb300 import learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows_off", [0, 3, -5])
@pytest.mark.parametrize("widths,batch", [((33, 33), 129), ((64, 64), 20000), ((704, 704), 5000), ((96, 40), 3000),
                                          ((24, 70), 3000), ((64, 64, 64), 5000)])
def test_outputs_over_inputs(pecs_lib, widths, batch, rows_off):
    """Many more tiles than the GPU runs at a time, so that a tile written early would be
    read by a later one."""
    torch = pytest.importorskip("torch")
    net = learned.Mlp(widths, seed=7)
    g = torch.Generator().manual_seed(batch)
    x = (2 * torch.rand((batch, widths[0]), generator=g) - 1).cuda()
    want = torch.empty((batch, widths[-1]), device="cuda")
    net.forward(x.data_ptr(), want.data_ptr(), batch)
    pad = 8 * max(widths)
    buf = torch.full((2 * pad + batch * max(widths),), float("nan"), device="cuda")
    for _ in range(3):
        buf[pad:pad + x.numel()] = x.flatten()
        torch.cuda.synchronize()
        y0 = pad + rows_off * widths[-1]
        net.forward(buf.data_ptr() + 4 * pad, buf.data_ptr() + 4 * y0, batch)
        assert torch.equal(buf[y0:y0 + want.numel()].view_as(want), want)
