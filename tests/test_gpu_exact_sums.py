"""The integer all-reduces of the grid-wide solvers: systems whose sums leave
their windows (one-iteration convergence, right-hand sides near the ends of
FP64's exponents, partials many orders apart), block counts at the edges of the
exchange, and reproducibility.  The systems have 9,000 to 20,000 rows, above
the cluster kernels' limit of 8,192."""
import numpy as np
import pytest

from _systems import pressure, unsymmetric

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system(orc):
    from fortranfvcell_gb300 import mesh
    return pressure(orc, mesh.square_mesh(101, 99, kind="quad", jitter=0.2, seed=3))


def _solve(s, code, b, tol, **kw):
    import torch
    from fortranfvcell_gb300 import Context
    from fortranfvcell_gb300.solver import make_opts
    c = Context()
    c.set_matrix(1, True, s["n"], s["nad"], s["ad"], s["au"], s["au"], s["ia"], s["ja"])
    x = torch.zeros(s["n"], dtype=torch.float64, device="cuda")
    st = c.solve(code, torch.from_numpy(b).cuda(), x, tol, 20000,
                 make_opts(kw.pop("precision", "fp64"), init=1, **kw))
    c.close()
    return x.cpu().numpy(), st


def _oracle(orc, s, code, b, tol):
    x = np.zeros(s["n"])
    rc, st = orc.solver(s["ad"].copy(), s["au"].copy(), s["au"].copy(), x, b.copy(), s["ia"],
                        s["ja"], s["n"], s["nad"], True, tol, 20000, code, 1)
    assert rc == 0
    return x, st


@pytest.mark.parametrize("scale", [1e-120, 1e-30, 1.0, 1e30, 1e120])
@pytest.mark.parametrize("code", [1, 2])
def test_scaled_right_hand_sides(orc, system, code, scale):
    """The stopping tests are relative for PCG; BiCGSTAB's compares a quotient
    with tol sqrt(|r.z|), so its tolerance follows the scale.  Bars as in the
    parity tests: 1e-10 (PCG), 1e-9 (BiCGSTAB) of the restated solver."""
    s = system if code == 1 else unsymmetric(system, seed=5)
    b = np.random.default_rng(11).uniform(-1.0, 1.0, s["n"])
    tol = 1e-10 if code == 1 else 1e-12
    want, so = _oracle(orc, s, code, b, tol)
    got, st = _solve(s, code, b * scale, tol if code == 1 else tol / scale)
    got = got / scale
    assert np.linalg.norm(got - want) <= (1e-10 if code == 1 else 1e-9) * np.linalg.norm(want)
    if code == 1:
        assert abs(st.iterations - so.iterations) <= 2


@pytest.mark.parametrize("code", [1, 2])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_one_iteration_convergence(system, code, precision):
    """A diagonal matrix: the first step solves it, and the sums drop to
    nothing (or exactly to zero) from one iteration to the next."""
    s = dict(system)
    s["au"] = np.zeros_like(system["au"])
    s["ad"] = np.random.default_rng(2).uniform(0.5, 2.0, s["n"])
    b = np.random.default_rng(3).uniform(-1.0, 1.0, s["n"])
    x, st = _solve(s, code, b, 1e-8, precision=precision)
    assert np.linalg.norm(s["ad"] * x - b) <= 1e-8 * np.linalg.norm(b)
    assert st.iterations <= 3


def test_partials_many_orders_apart(orc, system):
    """Right-hand side entries from 1e-200 to 1: most threads' partials lie
    below the window of the total."""
    b = 10.0 ** np.random.default_rng(7).uniform(-200, 0, system["n"])
    want, so = _oracle(orc, system, 1, b, 1e-10)
    got, st = _solve(system, 1, b, 1e-10)
    assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want)
    assert abs(st.iterations - so.iterations) <= 2


@pytest.mark.parametrize("kw", [dict(max_blocks=1), dict(max_blocks=2), dict(max_blocks=33),
                                dict(block_threads=128), dict(block_threads=384),
                                dict(block_threads=1024)])
@pytest.mark.parametrize("code", [1, 2])
def test_block_counts(orc, system, code, kw):
    s = system if code == 1 else unsymmetric(system, seed=5)
    b = np.random.default_rng(11).uniform(-1.0, 1.0, s["n"])
    tol = 1e-10 if code == 1 else 1e-12
    want, _ = _oracle(orc, s, code, b, tol)
    got, _ = _solve(s, code, b, tol, **kw)
    again, _ = _solve(s, code, b, tol, **kw)
    assert np.linalg.norm(got - want) <= (1e-10 if code == 1 else 1e-9) * np.linalg.norm(want)
    assert np.array_equal(got, again)


@pytest.mark.parametrize("kw", [dict(block_threads=128), dict(block_threads=256),
                                dict(max_blocks=1)])
def test_many_blocks(orc, kw):
    """More than 1024 blocks (128 threads): the counts of the words' top bits."""
    from fortranfvcell_gb300 import mesh
    s = pressure(orc, mesh.square_mesh(430, 430, kind="quad"))
    s = dict(s, au=-np.ones_like(s["au"]), ad=np.full(s["n"], 4.2))
    b = np.random.default_rng(11).uniform(-1.0, 1.0, s["n"])
    got, st = _solve(s, 1, b, 1e-12, **kw)
    want, so = _solve(s, 1, b, 1e-12)
    assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want)
    assert st.rel_residual <= 1e-9 and so.rel_residual <= 1e-9


def test_zero_and_nan_right_hand_sides(system):
    """b = 0: r.z = 0 and p.q = 0, the restated 0/0; a NaN ends the solve."""
    from fortranfvcell_gb300._lib import FVC_ERR_NAN, FvcError
    for bad in (0.0, np.nan, np.inf):
        b = np.zeros(system["n"])
        b[5] = bad
        with pytest.raises(FvcError) as e:
            _solve(system, 1, b, 1e-10)
        assert e.value.status == FVC_ERR_NAN
