"""The coarse cycle (k_coarse.cu) with fewer blocks than 16, as on a part of a
GPU, and without any: corrections bit-identical to separate launches; the cycle
runs in one launch where the blocks' shared memory holds the levels, and in none
with 0 blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _correction(name, over, prec, **tuning):
    import ugcore_gb300 as ug
    from ugcore_gb300 import problems
    ctx = ug.Context(0)
    ctx.set_tuning(**tuning)
    p = problems.Problem(ctx, problems.config(name, precision=prec, **over))
    d = ug.GPUVector(ctx, p.n).copy_from(np.random.default_rng(3).uniform(-1.0, 1.0, p.n))
    c = ug.GPUVector(ctx, p.n)
    p.gmg.apply(c, d)
    out = c.numpy()
    ctx.profile_begin()
    p.gmg.apply(c, d)
    prof = ctx.profile_end()
    assert np.array_equal(c.numpy(), out)
    return out, sum(n for k, (n, _) in prof.items() if "k_coarse_cycle" in k)


@pytest.mark.parametrize("name,over,prec", [("c3", dict(nref=5), "fp64"), ("c1", dict(nref=4), "fp64"),
                                            ("c1", dict(nref=4, mx=3, my=4, mz=2), "mixed"),
                                            ("c2", dict(nref=3, mx=5, my=5, mz=5), "fp64"),
                                            ("c2", dict(nref=4), "mixed")])
def test_bit_identical(name, over, prec):
    want, launches = _correction(name, over, prec, coarse_levels=0)
    assert launches == 0
    for blocks in (16, 8, 7, 4, 2, 1, 0):
        for levels in (-1, 3):
            got, launches = _correction(name, over, prec, coarse_blocks=blocks, coarse_levels=levels)
            assert np.array_equal(got, want), (blocks, levels)
            # (a few blocks' shared memory may not hold a base of 216 unknowns)
            assert launches == (1 if blocks else 0) or (levels == -1 or 0 < blocks < 8)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("over,launches", [
    (dict(mx=15, my=15, nref=2), 1), (dict(mx=16, my=15, nref=2), 0),       # bases of 256 and 272 rows
    (dict(mx=1, my=9, nref=3, nu1=4, nu2=4), 1), (dict(mx=3, my=3, nref=3, nu1=4, nu2=4), 1),   # one block
    (dict(mx=3, my=4, nref=4, nu1=4, nu2=4), 1)])                            # a cluster
def test_automatic_plans(over, launches, prec):
    over = dict(over, nu1=over.get("nu1", 1), nu2=over.get("nu2", 1))
    want, _ = _correction("c3", over, prec, coarse_levels=0)
    got, n = _correction("c3", over, prec)
    assert np.array_equal(got, want) and n == launches
