"""pecs_lu_solve_device_noalloc with other numbers of right-hand sides than the solve
that uploaded the factors: the upload loads the kernels of all of them (a kernel that is
first loaded at the call allocates device memory).  In a process of its own, where no
other test has loaded them."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

CODE = """
import ctypes as C
import numpy as np, scipy.sparse as sp, torch
import pecs_gb300 as pg
rng = np.random.default_rng(5)
n_cells = 300
A = sp.block_diag(list(rng.uniform(-1, 1, (n_cells, 2, 2)) + 3 * np.eye(2)), format="lil")
for i in range(n_cells - 1):
    A[2 * i, 2 * i + 2] = A[2 * i + 2, 2 * i] = 0.5
A = A.tocsr()
xy = np.stack([np.arange(n_cells) + 0.5, np.full(n_cells, 0.5)], axis=1)
for precision, tol in ((pg.PREC_FP64, 1e-12), (pg.PREC_FP32_IR, 1e-4)):
    lu = pg.LU(A, np.repeat(np.arange(n_cells, dtype=np.int32), 2), xy, precision=precision)
    b = torch.randn(8, A.shape[0], dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    lu.solve_device(b.data_ptr(), x.data_ptr(), nrhs=2)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for nrhs in range(1, 9):
        x.zero_()
        pg._ffi.check(pg.lib().pecs_lu_solve_device_noalloc(lu._h, nrhs, C.c_void_p(b.data_ptr()),
                                                            C.c_void_p(x.data_ptr()), C.c_void_p(0)))
        assert torch.cuda.mem_get_info()[0] == free, nrhs
        bh, xh = b[:nrhs].cpu().numpy(), x[:nrhs].cpu().numpy()
        assert np.linalg.norm((A @ xh.T).T - bh) < tol * np.linalg.norm(bh), nrhs
print("OK")
"""


def test_noalloc_with_other_numbers_of_right_hand_sides(pecs_lib):
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stdout + r.stderr
