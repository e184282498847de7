"""Host threads, each with its own context, that solve systems of different
sizes with the same kernel at once: the launches ask for different amounts of
shared memory (rows kept there), and every solve ends with the bits of the same
solve made alone."""
import threading

import numpy as np
import pytest

from test_gpu_staged import laplace_csrd, torch_dev

pytestmark = pytest.mark.gpu

SIZES = [(300, 301), (410, 409), (510, 511), (450, 447)]   # 90k to 261k rows


@pytest.mark.parametrize("code,precision", [(1, "fp64"), (2, "fp64"), (1, "mixed")])
def test_solves_of_different_sizes(code, precision):
    from fortranfvcell_gb300 import Context, make_opts
    opts = make_opts(precision, init=1, block_threads=1024)
    jobs = []
    for nx, ny in SIZES:
        s = laplace_csrd(nx, ny)
        c = Context()
        c.set_matrix(1, True, s["n"], s["nad"], s["ad"], s["au"], s["au"], s["ia"], s["ja"])
        b = torch_dev(np.random.default_rng(nx).uniform(-1, 1, s["n"]))
        x = torch_dev(np.zeros(s["n"]))

        def solve(c=c, b=b, x=x):
            return c.solve(code, b, x, 1e-300, 3, opts, raise_on_error=False).status
        status = solve()
        jobs.append((c, solve, x, status, x.cpu().numpy()))
    seen = [[] for _ in jobs]

    def loop(i):
        solve = jobs[i][1]
        for _ in range(300):
            seen[i].append(solve())
    threads = [threading.Thread(target=loop, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for got, (c, _, x, status, want) in zip(seen, jobs):
        assert got == [status] * 300
        assert np.array_equal(x.cpu().numpy(), want)
        c.close()
