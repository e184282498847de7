"""The blocks a batch of both solvers gives each system when the caller has no
hint: from the diagonal dominance of the BiCGSTAB systems' rows.  The batch
takes at most a quarter longer than with the iterations it is known to take as
hints, at every dominance (the shares are a guess of one number per system)."""
import numpy as np
import pytest

from test_gpu_staged import torch_dev

pytestmark = pytest.mark.gpu


def _grid(side, dom, seed):
    """CSRD arrays of a five-point matrix on side x (side + 1) cells: symmetric
    (dom None; lightly shifted), or couplings of 1 +- 0.4 with diagonals their
    absolute row sum plus the share dom."""
    nx, ny = side, side + 1
    n = nx * ny
    i = np.arange(n)
    x, y = i % nx, i // nx
    rows, cols = [], []
    for dx, dy in [(0, -1), (-1, 0), (1, 0), (0, 1)]:
        ok = (x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny)
        rows.append(i[ok])
        cols.append((i + dx + nx * dy)[ok])
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    order = np.lexsort((cols, rows))
    rows, cols = rows[order], cols[order]
    au = -np.ones(rows.size)
    if dom is not None:
        au *= 1.0 + 0.4 * np.random.default_rng(seed).uniform(-1, 1, au.size)
    ad = np.bincount(rows, np.abs(au), n) * (1.0 + (dom or 0.0)) + 1e-3
    ia = (np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]) + 1).astype(np.int32)
    return dict(ad=ad, au=au, ia=ia, ja=(cols + 1).astype(np.int32))


def _batch(sides, codes, dom):
    from fortranfvcell_gb300 import Context
    from fortranfvcell_gb300.solver import pack_block_diagonal
    systems = [_grid(side, dom if c == 2 else None, k)
               for k, (side, c) in enumerate(zip(sides, codes))]
    p = pack_block_diagonal(systems)
    ctx = Context()
    ctx.set_matrix(1, True, p["neq"], p["nad"], p["ad"], p["au"], p["au"], p["ia"], p["ja"])
    b = np.zeros(p["neq"])
    rng = np.random.default_rng(5)
    for r in p["rows"]:
        b[r] = rng.uniform(-1, 1, b[r].size)
    return ctx, p, torch_dev(b), torch_dev(np.zeros(p["neq"]))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("dom", [0.05, 0.0005, 0.0])
def test_shares_without_hints(precision, dom):
    from fortranfvcell_gb300 import make_opts
    sides = [int(round(100 * 2.8 ** ((7 * k % 24) / 23))) for k in range(24)]
    codes = [1 + k % 2 for k in range(24)]
    ctx, p, b, x = _batch(sides, codes, dom)
    tols = [1e-6 if c == 1 else 1e-9 for c in codes]
    opts = make_opts(precision, init=1)

    def run(hints):
        ms = []
        for _ in range(3):
            rc, st = ctx.solve_batched(p["row_start"], b, x, 0.0, 50000, opts, codes=codes,
                                       tols=tols, its_hint=hints)
            assert rc == 0
            ms.append(st[0].solve_ms)
        return min(ms), [float(s.iterations) for s in st]
    plain, its = run(None)
    hinted, _ = run(its)
    ctx.close()
    assert plain <= 1.25 * hinted, (plain, hinted)
