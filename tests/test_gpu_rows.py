"""Few-right-hand-side sweeps (rows.cu) where their tiles, teams and chunks have
edges: every width of a chunk of right-hand sides and one past it, a front whose
columns do not fit one staged chunk, nodes of one row, more children on a position
than a record holds, and solutions written over the right-hand sides."""
import numpy as np
import pytest
import scipy.sparse as sp

import pecs_gb300 as pg

pytestmark = pytest.mark.gpu


def _grid(nx, ny, b, seed):
    """Block five-point matrix, b unknowns per cell, diagonally dominant."""
    rng = np.random.default_rng(seed)
    n = nx * ny
    adj = sp.kron(sp.eye(ny), sp.diags([1.0, 1.0, 1.0], [-1, 0, 1], shape=(nx, nx))) + \
        sp.kron(sp.diags([1.0, 1.0], [-1, 1], shape=(ny, ny)), sp.eye(nx))
    A = sp.kron(adj, np.ones((b, b))).tocsr()
    A.data = rng.uniform(-1, 1, A.nnz)
    A = (A + 6 * b * sp.eye(n * b)).tocsr()
    xy = np.stack([np.tile(np.arange(nx), ny), np.repeat(np.arange(ny), nx)], 1) + 0.5
    return A, np.repeat(np.arange(n), b), xy, None


def _dense(n, seed):
    A = sp.csr_matrix(np.random.default_rng(seed).uniform(-1, 1, (n, n)) + n * np.eye(n))
    return A, np.zeros(n, int), np.array([[0.5, 0.5]]), None


def _arrow(cells, seed):
    """One dense cell coupled to `cells` class-0 cells: as many children on each of
    its positions."""
    rng = np.random.default_rng(seed)
    k, m = 3, 5
    n = cells * k + m
    A = np.zeros((n, n))
    for c in range(cells):
        s = slice(c * k, c * k + k)
        A[s, s] = rng.uniform(-1, 1, (k, k)) + 4 * np.eye(k)
        A[s, -m:] = rng.uniform(-1, 1, (k, m))
        A[-m:, s] = rng.uniform(-1, 1, (m, k))
    A[-m:, -m:] = rng.uniform(-1, 1, (m, m)) + 8 * cells * np.eye(m)
    cell = np.concatenate([np.repeat(np.arange(cells), k), np.full(m, cells)])
    xy = np.stack([np.arange(cells + 1) + 0.5, np.full(cells + 1, 0.5)], 1)
    cls = np.concatenate([np.zeros(cells * k, int), np.ones(m, int)])
    return sp.csr_matrix(A), cell, xy, cls


SYSTEMS = {"grid": lambda: _grid(13, 9, 5, 1), "one_row_nodes": lambda: _grid(21, 1, 1, 2),
           "one_cell": lambda: _dense(7, 3), "long_front": lambda: _dense(1100, 4),
           "many_children": lambda: _arrow(23, 5)}


@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 5, 6, 8, 9, 13, 17])
@pytest.mark.parametrize("name", SYSTEMS)
def test_solves_match_dense_elimination(pecs_lib, name, nrhs):
    """FP64 factors to 1e-12; FP32 factors to 1e-4, the residual a single sweep of
    single-precision values leaves on these diagonally dominant systems with room."""
    torch = pytest.importorskip("torch")
    A, cell, xy, cls = SYSTEMS[name]()
    n = A.shape[0]
    b = np.random.default_rng(nrhs).standard_normal((nrhs, n))
    ref = np.linalg.solve(A.toarray(), b.T).T
    for precision, tol in ((pg.PREC_FP64, 1e-12), (pg.PREC_FP32_IR, 1e-4)):
        lu = pg.LU(A, cell, xy, cls, precision=precision)
        x = lu.solve(b)
        assert np.linalg.norm(x - ref) < tol * np.linalg.norm(ref)
        d = torch.from_numpy(b).cuda()
        lu.solve_device(d.data_ptr(), d.data_ptr(), nrhs=nrhs)  # in place
        assert np.array_equal(d.cpu().numpy(), x)


@pytest.mark.parametrize("nrhs", [1, 3])
def test_tiles_of_several_chunks_with_update_rows(pecs_lib, nrhs):
    """A system large enough that forward tiles with update rows stage their values
    in chunks of fewer columns than the team has threads.  Relative residuals: the
    FP64 bound of the large-mesh tests (1e-10), FP32 values as above."""
    A, cell, xy, _ = _grid(128, 128, 8, 6)
    b = np.random.default_rng(nrhs).standard_normal((nrhs, A.shape[0]))
    for precision, tol in ((pg.PREC_FP64, 1e-10), (pg.PREC_FP32_IR, 1e-4)):
        x = pg.LU(A, cell, xy, precision=precision).solve(b)
        assert np.linalg.norm((A @ x.T).T - b) < tol * np.linalg.norm(b)
