"""pecs_warm_start_vectors (nn.cu) on both sides of the sizes from which it takes tiles:
few densities and coefficients (a thread per value) and many."""
import ctypes as C

import numpy as np
import pytest

import pecs_gb300 as pg

pytestmark = pytest.mark.gpu


def _call(torch, c, V, mean, nd, u_off):
    out = [torch.full((c.shape[0], nd), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
    p = lambda t: C.c_void_p(t.data_ptr())
    pg._ffi.check(pg.lib().pecs_warm_start_vectors(c.shape[0], c.shape[1], mean.numel() // 2, p(c), p(V), p(mean), nd,
                                                   u_off, p(out[0]), p(out[1]), C.c_void_p(0)))
    return out


@pytest.mark.parametrize("n_u,r", [(1, 1), (1, 33), (7, 3), (64, 32), (1000, 17), (1024, 31), (5000, 5), (9000, 40)])
@pytest.mark.parametrize("u_off", [0, 1, 300])
def test_rows_do_not_depend_on_the_batch(pecs_lib, n_u, r, u_off):
    """Each row of a batch that takes tiles (more than 2^18 densities, where r allows the
    other kernel) against the row by itself: the same bits.  Against FP64: r rounded
    multiply-adds of values below 8, exp to 2 ulp: 1e-5 relative with room."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n_u + r)
    nd = n_u + u_off + 13
    batch = min(3000, 2 ** 18 // (2 * n_u) + 3)
    t = lambda a: torch.from_numpy(a.astype(np.float32)).cuda()
    V, mean, c = t(rng.uniform(-1, 1, (2 * n_u, r))), t(rng.uniform(-2, 2, 2 * n_u)), t(rng.uniform(-1, 1, (batch, r)) / r ** 0.5)
    many = _call(torch, c, V, mean, nd, u_off)
    exact = torch.exp(mean.double() + c.double() @ V.double().T)
    for row in (0, batch // 2, batch - 1):
        one = _call(torch, c[row:row + 1].contiguous(), V, mean, nd, u_off)
        for k in range(2):
            assert torch.equal(one[k][0], many[k][row]), (row, k)
            want = torch.zeros(nd, dtype=torch.float64, device="cuda")
            want[u_off:u_off + n_u] = exact[row, k * n_u:(k + 1) * n_u]
            assert ((one[k][0] - want).abs() <= 1e-5 * want).all(), (row, k)
