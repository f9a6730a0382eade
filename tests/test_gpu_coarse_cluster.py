"""The coarse cycle over a cluster of blocks (k_coarse.cu) against separate
launches: bit-identical corrections where its levels are spread over the
blocks, where only the coarsest are left to the first one, with base levels of
a few to 216 rows, ragged parts, and the entry level just inside and outside
the automatic limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("c3", dict(nref=7), "fp64"), ("c3", dict(nref=6, mx=3, my=5), "mixed"), ("c0", dict(nref=6), "mixed"),
         ("c1", dict(nref=4), "fp64"), ("c1", dict(nref=4, mx=3, my=4, mz=2), "mixed"),
         ("c2", dict(nref=4), "mixed"), ("c2", dict(nref=3, mx=5, my=5, mz=5), "fp64"),
         ("c4", dict(nref=4), "mixed"), ("c4", dict(nref=3, mx=5, my=2, mz=3, nu1=1, nu2=3), "fp64")]


def _correction(levels, name, over, prec):
    import ugcore_gb300 as ug
    from ugcore_gb300 import problems
    ctx = ug.Context(0)
    ctx.set_tuning(coarse_levels=levels)
    p = problems.Problem(ctx, problems.config(name, precision=prec, **over))
    d = ug.GPUVector(ctx, p.n).copy_from(np.random.default_rng(3).uniform(-1.0, 1.0, p.n))
    c = ug.GPUVector(ctx, p.n)
    out = []
    for _ in range(2):
        p.gmg.apply(c, d)
        out.append(c.numpy())
    assert np.array_equal(out[0], out[1])
    return out[0]


@pytest.mark.parametrize("name,over,prec", CASES)
def test_bit_identical(name, over, prec):
    want = _correction(0, name, over, prec)
    for levels in (-1, 1, 2, 3, 4, 5, 7):
        assert np.array_equal(_correction(levels, name, over, prec), want), levels
