"""Mixed-precision CG with its row vectors kept in shared memory (the default
with 1024-thread blocks while a block's rows fit) against the plain-load kernel
of the same arithmetic (staging 1): the same iterates bit for bit, also where a
solve stops with an odd or an even number of iterations since its last residual
replacement."""
import numpy as np
import pytest

from test_gpu_staged import laplace_csrd, torch_dev

pytestmark = pytest.mark.gpu


def _both(s, b, tol, maxit):
    from fortranfvcell_gb300 import Context, make_opts
    ctx = Context()
    ctx.set_matrix(1, True, s["n"], s["nad"], s["ad"], s["au"], s["au"], s["ia"], s["ja"])
    out = []
    for staging in (0, 1):
        bd, xd = torch_dev(b), torch_dev(np.zeros(s["n"]))
        st = ctx.solve(1, bd, xd, tol, maxit,
                       make_opts("mixed", init=1, staging=staging, block_threads=1024),
                       raise_on_error=False)
        out.append((st.status, st.inner_iterations, st.iterations, xd.cpu().numpy()))
    ctx.close()
    return out


# one slice and less, one block to its edge and beyond it, 16-bit offsets
# exceeded (no uniform layout), two rows per thread
@pytest.mark.parametrize("nx,ny", [(7, 3), (32, 32), (41, 25), (97, 53), (40000, 3), (420, 421)])
@pytest.mark.parametrize("tol,maxit", [(1e-9, 20000), (1e-300, 37), (1e-300, 38)])
def test_kept_matches_plain(nx, ny, tol, maxit):
    s = laplace_csrd(nx, ny)
    b = np.random.default_rng(4).uniform(-1, 1, s["n"])
    kept, plain = _both(s, b, tol, maxit)
    assert kept[:3] == plain[:3]
    assert np.array_equal(kept[3], plain[3])


@pytest.mark.parametrize("kind", ["tri", "mixed"])
def test_kept_matches_plain_on_mesh(kind):
    # a pinned row, frozen in the FP32 iteration; triangles: slices of three
    from fortranfvcell_gb300 import mesh
    p = mesh.pressure_system(mesh.square_mesh(300, kind=kind, jitter=0.2, seed=5), matriz=1,
                             unsym=True, pin_cell=1)
    s = dict(n=p.neq, nad=p.nad, ad=p.ad, au=p.au, ia=p.ia, ja=p.ja)
    b = np.random.default_rng(6).uniform(-1, 1, p.neq)
    kept, plain = _both(s, b, 1e-8, 50000)
    assert kept[:3] == plain[:3] and kept[0] == 0
    assert np.array_equal(kept[3], plain[3])
