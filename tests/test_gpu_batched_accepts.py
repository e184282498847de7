"""Batches that the automatic shape takes whatever limits the caller sets: more
systems than one launch of groups holds under max_blocks, blocks_per_sm or large
blocks go to clusters, which have no such bound."""
import numpy as np
import pytest

from test_gpu_batched_shares import _batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nsys,kw", [(700, dict(max_blocks=650)), (700, dict(blocks_per_sm=4)),
                                     (700, dict(block_threads=1024)), (1100, dict()),
                                     (1300, dict())])
def test_more_systems_than_groups_hold(precision, nsys, kw):
    """The recomputed residuals are within ten times the tolerance of the
    recurrence's."""
    from fortranfvcell_gb300 import make_opts
    ctx, p, b, x = _batch([6] * nsys, [2] * nsys, 0.05)
    rc, st = ctx.solve_batched(p["row_start"], b, x, 1e-9, 2000,
                               make_opts(precision, init=1, stop_rule=1, **kw),
                               codes=[2] * nsys)
    assert rc == 0
    assert max(s.rel_residual for s in st) <= 1e-8
    ctx.close()
    assert np.isfinite(x.cpu().numpy()).all()
