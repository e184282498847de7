"""The cell kernels with the geometry cache against the same kernels without
it, bit for bit, where the division through a cached reciprocal changes over to
the plain division: meshes scaled towards the ends of FP64's exponents, zero
fields (zero dividends), two materials.  And gradient calls from more threads
than there are error words."""
import numpy as np
import pytest

from test_gpu_cells import dev, fields, host, random_case

pytestmark = pytest.mark.gpu


def _momentum(case, f, cached):
    from fortranfvcell_gb300 import cells
    m = cells.CellMesh(case["coor"], case["ix"], case["nelcon"], case["num"], case["pedge"],
                       case["sedge"], case["e"])
    if cached:
        m.cache_geometry()
    n, nsh = case["numel"], case["nshared"]
    ad, b, res = (dev(np.zeros(n)) for _ in range(3))
    au, im, d = dev(np.zeros(nsh * n)), dev(np.zeros((n, 4))), dev(np.zeros((n, 2)))
    ia = dev(np.array([nsh, 0], np.int32))
    cells.momentum(m, 1, 1, dev(f["u1"]), dev(f["p"]), dev(f["w"]), dev(f["g1"]), dev(f["g2"]),
                   dev(f["gp"]), 0.05, ia, ia, 4, ad, au, b, im, d, res, under_u=0.7)
    return [host(t) for t in (ad, au, b, im, d, res)]


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -390, 2.0 ** -402, 2.0 ** 390, 2.0 ** 402])
@pytest.mark.parametrize("field", [0.0, 1.0, 1e-110])
def test_division_through_reciprocal(orc, scale, field):
    case, rng = random_case(orc, "mixed", 8, 3)
    case["coor"] = case["coor"] * scale
    f = {k: v * field for k, v in fields(rng, case["numel"]).items()}
    for got, want in zip(_momentum(case, f, True), _momentum(case, f, False)):
        assert np.array_equal(got, want, equal_nan=True)


def test_more_gradient_calls_than_error_words(orc):
    import threading

    import torch
    from fortranfvcell_gb300 import FvcError, cells
    case, rng = random_case(orc, "quad", 9, 1)
    f = fields(rng, case["numel"])
    bad = dict(case, pedge=np.where(case["pedge"] == 4, 7, case["pedge"]).astype(np.int32))
    m, mb = (cells.CellMesh(c["coor"], c["ix"], c["nelcon"], c["num"], c["pedge"], c["sedge"],
                            c["e"]) for c in (case, bad))
    assert (case["pedge"] == 4).any()
    out, want = {}, dev(np.zeros((case["numel"], 2)))
    cells.gradient(m, 1, 1, dev(f["u1"]), want)
    u = dev(f["u1"])
    grads = [dev(np.zeros((case["numel"], 2))) for _ in range(80)]
    torch.cuda.synchronize()

    def call(i):
        for _ in range(5):
            try:
                cells.gradient(mb if i % 2 else m, 1, 1, u, grads[i])
                out.setdefault(i, []).append(True)
            except FvcError:
                out.setdefault(i, []).append(False)
    threads = [threading.Thread(target=call, args=(i,)) for i in range(80)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(80):
        assert out[i] == [i % 2 == 0] * 5
        if i % 2 == 0:
            assert np.array_equal(host(grads[i]), host(want))
