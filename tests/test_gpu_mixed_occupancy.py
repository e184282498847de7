"""Blocks of 128 and 256 threads of the plain-load mixed CG lie two on an SM, beside
a first-level cache left near its largest: on rows that fill them, a fifth or more
faster than one an SM (they are bound by loads in flight; one an SM is what a
block's shared memory left when the kernel's had outgrown the cache's split)."""
import numpy as np
import pytest

from test_gpu_batched_shares import _grid
from test_gpu_staged import torch_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [128, 256])
def test_two_blocks_on_an_sm(threads):
    from fortranfvcell_gb300 import Context, make_opts
    s = _grid(1000, None, 1)
    n = s["ad"].size
    ctx = Context()
    ctx.set_matrix(1, True, n, s["ja"].size, s["ad"], s["au"], s["au"], s["ia"], s["ja"])
    b, x = torch_dev(np.random.default_rng(4).uniform(-1, 1, n)), torch_dev(np.zeros(n))

    def ms(**kw):
        o = make_opts("mixed", init=1, block_threads=threads, **kw)
        return min(ctx.solve(1, b, x, 1e-300, 40, o, raise_on_error=False).solve_ms
                   for _ in range(4))
    two, one = ms(), ms(blocks_per_sm=1)
    ctx.close()
    assert two <= 0.85 * one, (two, one)
