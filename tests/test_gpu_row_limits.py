"""The sizes at which the solvers change what they keep of a row: the mixed CG's
kept form at three, five and seven rows per thread and the first size of the
staged form; the FP64 CG on both sides of the size from which its sums keep an
order, and of the block size up to which x is updated under a sum."""
import numpy as np
import pytest

from test_gpu_batched_shares import _grid
from test_gpu_staged import laplace_csrd, torch_dev

pytestmark = pytest.mark.gpu

def _context(s):
    from fortranfvcell_gb300 import Context
    c = Context()
    c.set_matrix(1, True, s["ad"].size, s["ja"].size, s["ad"], s["au"], s["au"], s["ia"], s["ja"])
    return c


@pytest.mark.parametrize("side,rows", [(640, 3), (850, 5), (1020, 7), (1043, 7), (1046, 8)])
def test_kept_and_staged_match_plain(side, rows):
    """The same iterates bit for bit as the plain-load kernel, with an odd and an
    even number of iterations since the last residual replacement."""
    from fortranfvcell_gb300 import make_opts
    s = _grid(side, None, 1)
    n = s["ad"].size
    slices = -(-n // 32)
    assert -(-(-(-slices // 152)) // 32) == rows      # 152 SMs, 32 warps each
    b = np.random.default_rng(4).uniform(-1, 1, n)
    ctx = _context(s)
    for maxit in (37, 38):
        out = []
        for staging in (0, 1):
            bd, xd = torch_dev(b), torch_dev(np.zeros(n))
            st = ctx.solve(1, bd, xd, 1e-300, maxit,
                           make_opts("mixed", init=1, staging=staging, block_threads=1024),
                           raise_on_error=False)
            out.append((st.status, st.inner_iterations, st.iterations, xd.cpu().numpy()))
        assert out[0][:3] == out[1][:3]
        assert np.array_equal(out[0][3], out[1][3])
    ctx.close()


def _dominant(s):
    """The five-point matrix s with its shift taken out and its diagonal 5 % up."""
    return dict(s, ad=1.05 * (s["ad"] - 1e-3))


def _solve_known(s, **kw):
    """The error of a solve whose solution is known.  The matrix is symmetric and
    5 % dominant with row sums of 2 to 4: |A| |A^-1| is below 2.05 / 0.05 times 2,
    and a residual reduced by 1e-13 leaves an error below 1e-11."""
    from fortranfvcell_gb300 import make_opts
    n = s["ad"].size
    rows = np.repeat(np.arange(n), np.diff(s["ia"]))
    x = np.random.default_rng(3).uniform(-1, 1, n)
    b = s["ad"] * x + np.bincount(rows, s["au"] * x[s["ja"] - 1], n)
    ctx = _context(s)
    got = torch_dev(np.zeros(n))
    ctx.solve(1, torch_dev(b), got, 1e-13, 500, make_opts("fp64", init=1, stop_rule=1, **kw))
    ctx.close()
    return np.linalg.norm(got.cpu().numpy() - x) / np.linalg.norm(x)


# 523,452 and 524,900 rows (ordered sums from 524,288 on)
@pytest.mark.parametrize("side", [723, 724])
def test_ordered_sums(side):
    s = _dominant(_grid(side, None, 1))
    assert (s["ad"].size >= 524288) == (side == 724)
    assert _solve_known(s) <= 1e-11


# one block of 32 warps: ten slices to each, one more, eleven to each
@pytest.mark.parametrize("nx,ny,slices", [(80, 128, 320), (95, 108, 321), (88, 128, 352)])
@pytest.mark.parametrize("max_blocks", [1, 2])
def test_late_x(nx, ny, slices, max_blocks):
    s = _dominant(laplace_csrd(nx, ny))
    assert -(-s["ad"].size // 32) == slices
    assert _solve_known(s, max_blocks=max_blocks, block_threads=1024) <= 1e-11
