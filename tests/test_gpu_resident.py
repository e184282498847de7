"""The rows a grid-wide solver keeps in shared memory: none, some and all of a
thread's rows (one, two and eight blocks over 12,120 rows), rows of more
entries than are kept, the transposed product, and BiCGSTAB on both sides of
the size from which its z vectors are stored.  The matrices are 5 %
diagonally dominant with diagonals of 2 to 11, so |A| |A^-1| is below 250 and a
residual reduced by 1e-13 leaves an error below 3e-11 of x; the bar is 1e-10
against a direct solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(nx, ny, wide, unsym, seed=1):
    """CSRD arrays of a five-point matrix, with diagonal neighbours too in the
    upper half of the rows (wide), and the same as a scipy matrix."""
    import scipy.sparse as sp
    n = nx * ny
    i = np.arange(n)
    x, y = i % nx, i // nx
    rows, cols = [], []
    for dx, dy in [(0, -1), (-1, 0), (1, 0), (0, 1), (-1, -1), (1, -1), (-1, 1), (1, 1)]:
        ok = (x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny)
        j = i + dx + nx * dy
        if dx and dy:
            ok &= (i >= n // 2) & (j >= n // 2)
            if not wide:
                ok &= False
        rows.append(i[ok])
        cols.append(j[ok])
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    order = np.lexsort((cols, rows))
    rows, cols = rows[order], cols[order]
    rng = np.random.default_rng(seed)
    au = -np.ones(rows.size)
    if unsym:
        au *= 1.0 + 0.4 * rng.uniform(-1, 1, au.size)
    off = sp.csr_matrix((au, (rows, cols)), shape=(n, n))
    ad = 1.05 * np.asarray(np.maximum(abs(off).sum(axis=1).ravel(), abs(off).sum(axis=0).ravel())).ravel()
    ia = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32) + 1
    return n, ad, au, ia, (cols + 1).astype(np.int32), (off + sp.diags(ad)).tocsc()


def _check(nx, ny, wide, how, **kw):
    import torch
    from scipy.sparse.linalg import spsolve
    from fortranfvcell_gb300 import Context
    from fortranfvcell_gb300.solver import make_opts
    n, ad, au, ia, ja, full = _matrix(nx, ny, wide, how != "pcg")
    b = np.random.default_rng(2).uniform(-1.0, 1.0, n)
    want = spsolve(full.T.tocsc() if how == "transposed" else full, b)
    c = Context()
    c.set_matrix(1, True, n, ja.size, ad, au, au, ia, ja)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    o = make_opts("fp64", init=1, stop_rule=1, **kw)
    if how == "transposed":
        c.solve_transposed(torch.from_numpy(b).cuda(), x, 1e-13, 1000, o)
    else:
        c.solve(1 if how == "pcg" else 2, torch.from_numpy(b).cuda(), x, 1e-13, 1000, o)
    c.close()
    got = x.cpu().numpy()
    assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want)


@pytest.mark.parametrize("how", ["pcg", "bicgstab", "transposed"])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("max_blocks", [1, 2, 8])
def test_rows_kept(how, wide, max_blocks):
    _check(120, 101, wide, how, max_blocks=max_blocks)


@pytest.mark.parametrize("how", ["bicgstab", "transposed"])
@pytest.mark.parametrize("nx,ny", [(255, 257), (256, 257)])
@pytest.mark.parametrize("max_blocks", [0, 5])
def test_stored_z(how, nx, ny, max_blocks):
    _check(nx, ny, True, how, max_blocks=max_blocks)
