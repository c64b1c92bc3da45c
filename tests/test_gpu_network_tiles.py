"""Forward passes of the network (nn.cu) with tiles of 32, 64 and 128 columns: the batch and
the layer's width choose, at the counts of tiles where the choice changes and at widths
that are no whole tile."""
import pytest

from pecs_gb300 import learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths", [(5, 33), (40, 65, 3), (64, 129, 100), (65, 704, 72), (7, 2049, 64), (130, 128)])
@pytest.mark.parametrize("batch", [257, 1000, 1153, 2432, 19457])
def test_rows_do_not_depend_on_the_batch(pecs_lib, widths, batch):
    """The first, last and middle rows of a batch against batches of 40 of them: the same bits,
    whatever the tile.  Against FP64 sums of the BF16-rounded operands: 16 terms of the
    tensor core's own sums at a time, FP32 in between, 2^-22 times the sum of the terms'
    sizes; a hidden value that this moves across a BF16 rounding (2^-9 of at most one)
    moves an output by that times its weight, few of them: 1e-2 of the largest output."""
    torch = pytest.importorskip("torch")
    net = learned.Mlp(widths, seed=3)
    x = (2 * torch.rand((batch, widths[0]), generator=torch.Generator().manual_seed(batch)) - 1).cuda()
    y = torch.empty((batch, widths[-1]), device="cuda")
    net.forward(x.data_ptr(), y.data_ptr(), batch)
    p = torch.from_numpy(net.get_params()).double()
    for lo in (0, batch // 2, batch - 40):
        part = x[lo:lo + 40].contiguous()
        few = torch.empty((40, widths[-1]), device="cuda")
        net.forward(part.data_ptr(), few.data_ptr(), 40)
        assert torch.equal(few, y[lo:lo + 40]), lo
        h, off = part.cpu().double(), 0
        for l, (k, n) in enumerate(zip(widths[:-1], widths[1:])):
            W, b = p[off:off + k * n].view(n, k), p[off + k * n:off + k * n + n]
            off += k * n + n
            h = h.float().bfloat16().double() @ W.float().bfloat16().double().T + b
            if l + 2 < len(widths):
                h = torch.tanh(h)
        assert (few.cpu().double() - h).abs().max() < 1e-2 * h.abs().max(), lo
