"""Few-right-hand-side solves (rows.cu) of systems with levels of short teams and long
rows: many class-0 cells of a few unknowns, all of them coupled to one dense cell.  A
team's source values are then staged a part of a row at a time so that the teams of a
CTA fit its shared memory."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg

import pecs_gb300 as pg

pytestmark = pytest.mark.gpu


def _bordered(cells, k, m, seed):
    rng = np.random.default_rng(seed)
    n = cells * k + m
    D = sp.block_diag(list(rng.uniform(-1, 1, (cells, k, k)) + 4 * np.eye(k) * np.sqrt(m)), format="csr")
    B, C = rng.uniform(-1, 1, (cells * k, m)), rng.uniform(-1, 1, (m, cells * k))
    E = rng.uniform(-1, 1, (m, m)) + 4 * n * np.eye(m)
    A = sp.bmat([[D, sp.csr_matrix(B)], [sp.csr_matrix(C), sp.csr_matrix(E)]], format="csr")
    cell = np.concatenate([np.repeat(np.arange(cells), k), np.full(m, cells)])
    xy = np.stack([np.arange(cells + 1) + 0.5, np.full(cells + 1, 0.5)], 1)
    cls = np.concatenate([np.zeros(cells * k, int), np.ones(m, int)])
    return A, cell, xy, cls, (D, B, C, E)


def _exact(parts, b):
    """Block elimination: x of [D B; C E] x = b for the columns of b."""
    D, B, C, E = parts
    k = D.shape[0]
    lu = sp.linalg.splu(D.tocsc())
    x2 = np.linalg.solve(E - C @ lu.solve(B), b[k:] - C @ lu.solve(b[:k]))
    return np.concatenate([lu.solve(b[:k] - B @ x2), x2])


@pytest.mark.parametrize("cells,k,m", [(2500, 3, 380), (3000, 2, 450), (3000, 3, 500)])
def test_long_rows_among_small_nodes(pecs_lib, cells, k, m):
    """Every chunk of right-hand sides that the factors are applied to.  FP64 to 1e-12,
    FP32 factors to 1e-4 of block elimination: the bounds of the other direct solves of
    diagonally dominant systems."""
    torch = pytest.importorskip("torch")
    A, cell, xy, cls, parts = _bordered(cells, k, m, 1)
    b = np.random.default_rng(2).standard_normal((17, A.shape[0]))
    ref = _exact(parts, b.T).T
    for precision, tol in ((pg.PREC_FP64, 1e-12), (pg.PREC_FP32_IR, 1e-4)):
        lu = pg.LU(A, cell, xy, cls, precision=precision)
        for nrhs in (1, 2, 3, 4, 5, 6, 8, 12, 16, 17):
            x = lu.solve(b[:nrhs])
            assert np.linalg.norm(x - ref[:nrhs]) < tol * np.linalg.norm(ref[:nrhs]), (precision, nrhs)
            d = torch.from_numpy(b[:nrhs]).cuda()
            lu.solve_device(d.data_ptr(), d.data_ptr(), nrhs=nrhs)  # in place
            assert np.array_equal(d.cpu().numpy(), x), (precision, nrhs)
