"""How full a batch's groups of blocks fill the device: the automatic shape takes
at most a fifth longer than the better of the full ones (128-thread blocks eight
to an SM, 256-thread blocks four), with few large systems as with many small
ones.  cluster_size 1: groups (64 mixed systems of 128^2 would go to clusters)."""
import numpy as np
import pytest

from test_gpu_batched_shares import _batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nsys,side", [(64, 128), (16, 256), (8, 400), (32, 48), (48, 100)])
def test_automatic_shape(precision, nsys, side):
    from fortranfvcell_gb300 import make_opts
    codes = [1] * nsys
    ctx, p, b, x = _batch([side] * nsys, codes, 0.0)

    def ms(**kw):
        opts = make_opts(precision, init=1, cluster_size=1, **kw)
        best = np.inf
        for _ in range(4):
            rc, st = ctx.solve_batched(p["row_start"], b, x, 1e-6, 50000, opts, codes=codes)
            assert rc == 0
            best = min(best, st[0].solve_ms)
        return best
    auto = ms()
    full = min(ms(block_threads=128, blocks_per_sm=8),
               ms(block_threads=256, blocks_per_sm=4))
    ctx.close()
    assert auto <= 1.2 * full, (auto, full)
