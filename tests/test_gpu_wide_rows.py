"""Rows of more than four off-diagonals, which the row sums take four entries
at a time: every remainder, in the products (the reference's rounding bit for
bit, the fused and the FP32 form within their rounding) and in the solvers that
share them, transposed and mixed too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WIDTHS = [1, 4, 5, 6, 7, 8, 9, 12, 13]


def _pattern(n, width):
    """A symmetric pattern of `width` off-diagonals in the inner rows: bands in
    pairs and, for an odd width, each row's partner 512 rows away."""
    i = np.arange(n)
    offs = []
    for d in (1, 97, 3, 211, 5, 301)[: width // 2]:
        offs += [d, -d]
    rows, cols = [], []
    for d in offs:
        ok = (i + d >= 0) & (i + d < n)
        rows.append(i[ok])
        cols.append((i + d)[ok])
    if width % 2:
        ok = (i ^ 512) < n
        rows.append(i[ok])
        cols.append((i ^ 512)[ok])
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    order = np.lexsort((cols, rows))
    return rows[order], cols[order]


def _csrd(n, width, seed=1, unsym=True):
    """CSRD arrays, 5 % diagonally dominant by rows and by columns."""
    rows, cols = _pattern(n, width)
    rng = np.random.default_rng(seed)
    au = -np.ones(rows.size)
    if unsym:
        au *= 1.0 + 0.4 * rng.uniform(-1, 1, au.size)
    ad = 1.05 * np.maximum(np.bincount(rows, np.abs(au), n), np.bincount(cols, np.abs(au), n))
    ia = (np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]) + 1).astype(np.int32)
    return dict(n=n, ad=ad, au=au, ia=ia, ja=(cols + 1).astype(np.int32), rows=rows, cols=cols)


def _context(s):
    from fortranfvcell_gb300 import Context
    c = Context()
    c.set_matrix(1, True, s["n"], s["ja"].size, s["ad"], s["au"], s["au"], s["ia"], s["ja"])
    return c


def _product(s, x):
    """The row sums in the reference's order, each product and sum rounded."""
    y = s["ad"] * x
    k = np.arange(s["ja"].size) - (s["ia"][s["rows"]] - 1)
    for j in range(int(k.max()) + 1):
        m = k == j
        y[s["rows"][m]] += s["au"][m] * x[s["cols"][m]]
    return y


@pytest.mark.parametrize("width", WIDTHS)
def test_products(width):
    import torch
    s = _csrd(3001, width)
    x = np.random.default_rng(3).uniform(-1, 1, s["n"])
    want = _product(s, x)
    c = _context(s)
    xd = torch.from_numpy(x).cuda()
    y = torch.empty_like(xd)
    c.spmv(xd, y)
    assert np.array_equal(y.cpu().numpy(), want)
    # both sums round each of their width + 1 terms at most twice
    scale = np.abs(s["ad"] * x) + np.bincount(s["rows"], np.abs(s["au"] * x[s["cols"]]), s["n"])
    c.spmv_fast(xd, y)
    assert (np.abs(y.cpu().numpy() - want) <= 4 * (width + 1) * 2.0 ** -53 * scale).all()
    # FP32, as row sums of (excess, couplings): weights, differences and terms
    # are rounded to 24 bits
    x3 = torch.from_numpy(x.astype(np.float32)).cuda()
    y3 = torch.empty_like(x3)
    c.spmv_f32(x3, y3)
    c.close()
    assert (np.abs(y3.cpu().numpy() - want) <= 8 * (width + 3) * 2.0 ** -24 * 2 * scale + 1e-30).all()


@pytest.mark.parametrize("width", [5, 6, 7, 9, 13])
@pytest.mark.parametrize("how", ["pcg", "bicgstab", "transposed", "mixed pcg", "mixed bicgstab"])
def test_solves(width, how):
    """|A| |A^-1| is below 2.05 / 0.05 times the ratio of the largest to the
    smallest row sum (4.7: half the entries, each 1 +- 0.4), and the residuals
    are reduced by 1e-12: the error is below 1e-9 of x."""
    import scipy.sparse as sp
    import torch
    from scipy.sparse.linalg import spsolve
    from fortranfvcell_gb300 import make_opts
    s = _csrd(9001, width, unsym="pcg" not in how)
    n = s["n"]
    full = (sp.csr_matrix((s["au"], (s["rows"], s["cols"])), shape=(n, n)) + sp.diags(s["ad"])).tocsc()
    b = np.random.default_rng(2).uniform(-1.0, 1.0, n)
    want = spsolve(full.T.tocsc() if how == "transposed" else full, b)
    c = _context(s)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    o = make_opts("mixed" if "mixed" in how else "fp64", init=1, stop_rule=1)
    bd = torch.from_numpy(b).cuda()
    if how == "transposed":
        c.solve_transposed(bd, x, 1e-12, 1000, o)
    else:
        c.solve(1 if "pcg" in how else 2, bd, x, 1e-12, 1000, o)
    c.close()
    assert np.linalg.norm(x.cpu().numpy() - want) <= 1e-9 * np.linalg.norm(want)


@pytest.mark.parametrize("width", [4, 6])
@pytest.mark.parametrize("slices", [24575, 24576, 24577])
@pytest.mark.parametrize("ragged", [0, 31])
def test_products_of_many_slices(width, slices, ragged):
    """Both sides of the size from which narrow rows are summed in fewer
    registers, the last slice full or of one row; bars as above."""
    import torch
    s = _csrd(32 * slices - ragged, width)
    x = np.random.default_rng(3).uniform(-1, 1, s["n"])
    want = _product(s, x)
    c = _context(s)
    xd = torch.from_numpy(x).cuda()
    y = torch.empty_like(xd)
    c.spmv(xd, y)
    assert np.array_equal(y.cpu().numpy(), want)
    c.spmv_fast(xd, y)
    c.close()
    scale = np.abs(s["ad"] * x) + np.bincount(s["rows"], np.abs(s["au"] * x[s["cols"]]), s["n"])
    assert (np.abs(y.cpu().numpy() - want) <= 4 * (width + 1) * 2.0 ** -53 * scale).all()
