"""The windows of the exact sums of FP32 pairs: the mixed BiCGSTAB of a weakly
dominant matrix, whose products cancel (partials far above their total), against
a strongly dominant one of the same size.  Its iteration does the same work, with
fewer FP64 residual sweeps among its iterations, so that it takes no longer;
sums that leave their window are taken again and cost it half as much again or
more.  The bar leaves 15 % for the timing."""
import numpy as np
import pytest

from test_gpu_staged import laplace_csrd, torch_dev

pytestmark = pytest.mark.gpu


def _system(nx, ny, dom, seed=1):
    s = laplace_csrd(nx, ny)
    rows = np.repeat(np.arange(s["n"]), np.diff(s["ia"]))
    s["au"] = s["au"] * (1.0 + 0.4 * np.random.default_rng(seed).uniform(-1, 1, s["nad"]))
    s["ad"] = np.bincount(rows, np.abs(s["au"]), s["n"]) * (1.0 + dom) + 1e-3
    return s


def _us_per_iteration(s):
    from fortranfvcell_gb300 import Context, make_opts
    ctx = Context()
    ctx.set_matrix(1, True, s["n"], s["nad"], s["ad"], s["au"], s["au"], s["ia"], s["ja"])
    b, x = torch_dev(np.random.default_rng(4).uniform(-1, 1, s["n"])), torch_dev(np.zeros(s["n"]))
    best, its = np.inf, 0
    for _ in range(6):
        st = ctx.solve(2, b, x, 1e-7, 20000, make_opts("mixed", init=1))
        its = st.inner_iterations
        best = min(best, 1e3 * st.solve_ms / its)
    ctx.close()
    return best, its


@pytest.mark.parametrize("nx,ny", [(25, 24), (55, 54), (131, 130)])
def test_cancelling_products(nx, ny):
    easy, its_easy = _us_per_iteration(_system(nx, ny, 0.05))
    hard, its_hard = _us_per_iteration(_system(nx, ny, 0.0))
    assert its_hard > 3 * its_easy
    assert hard <= 1.15 * easy, (hard, easy)


@pytest.mark.parametrize("nx,ny", [(45, 46), (110, 109)])
@pytest.mark.parametrize("code", [1, 2])
@pytest.mark.parametrize("scale", [1e-130, 1e130])
def test_sums_near_the_ends_of_the_exponents(nx, ny, code, scale):
    """Totals of 1e-260 and 1e260 have windows like any other: an iteration takes
    as long as with totals of 1e-200 (a tenth for the timing)."""
    from fortranfvcell_gb300 import Context, make_opts
    s = _system(nx, ny, 0.05)
    ctx = Context()
    ctx.set_matrix(1, True, s["n"], s["nad"], s["ad"], s["au"], s["au"], s["ia"], s["ja"])
    b, us = np.random.default_rng(4).uniform(-1, 1, s["n"]), []
    for sc in (1e-100, scale):
        bd, x, best = torch_dev(b * sc), torch_dev(np.zeros(s["n"])), np.inf
        for _ in range(6):
            st = ctx.solve(code, bd, x, 0.0, 25, make_opts("fp64", init=1), raise_on_error=False)
            assert st.iterations == 25
            best = min(best, st.solve_ms)
        us.append(best)
    ctx.close()
    assert us[1] <= 1.1 * us[0], us
