"""Right-hand sides so small that the sums of the recurrence are subnormal: they
are rounded like any other FP64 sum, and the solve ends at about the residual of
the same system at scale 1.  The sums of 9,999 rows at 1e-157 are 1e-310, 44 bits
of the subnormals' grid, and fall by 1e-6 or so until the tolerance: 24 bits are
left, so the residual is allowed twice that of the other solve."""
import numpy as np
import pytest

from _systems import pressure, unsymmetric

pytestmark = pytest.mark.gpu


def _residuals(orc, side, code, tol, scales):
    """|b - A x| / |b| of the solves of the right-hand sides b * scale."""
    import scipy.sparse as sp
    import torch
    from fortranfvcell_gb300 import Context, mesh
    from fortranfvcell_gb300.solver import make_opts
    s = pressure(orc, mesh.square_mesh(side, side + 2, kind="quad", jitter=0.2, seed=3))
    if code == 2:
        s = unsymmetric(s, seed=5)
    n = s["n"]
    rows = np.repeat(np.arange(n), np.diff(s["ia"]))
    full = sp.csr_matrix((s["au"][:rows.size], (rows, s["ja"][:rows.size] - 1)), shape=(n, n))
    full = full + sp.diags(s["ad"])
    b = np.random.default_rng(11).uniform(-1.0, 1.0, n)
    c = Context()
    c.set_matrix(1, True, n, s["nad"], s["ad"], s["au"], s["au"], s["ia"], s["ja"])
    out = []
    for scale in scales:
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        c.solve(code, torch.from_numpy(b * scale).cuda(), x, tol, 5000,
                make_opts("fp64", init=1, stop_rule=1))
        out.append(np.linalg.norm(b - full @ (x.cpu().numpy() / scale)) / np.linalg.norm(b))
    c.close()
    return out


@pytest.mark.parametrize("side", [40, 99])       # one cluster (PCG); the whole grid
@pytest.mark.parametrize("code", [1, 2])
def test_subnormal_sums(orc, side, code):
    want, got = _residuals(orc, side, code, 1e-3, [1.0, 1e-157])
    assert got <= 2.0 * want, (got, want)


@pytest.mark.parametrize("side", [40, 99])
@pytest.mark.parametrize("code", [1, 2])
def test_sums_that_become_subnormal(orc, side, code):
    """At 1e-150 the sums reach the subnormals as the solve converges: to the
    tolerance, as at scale 1 (the recurrence's residual within a tenth)."""
    got, = _residuals(orc, side, code, 1e-6, [1e-150])
    assert got <= 1.1e-6, got
