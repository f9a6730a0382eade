"""Small 3D FP32 levels with their smoothing in two launches (k_level3d.cu)
against the step-by-step kernels of the SELL format: the same row operations in
the same order, so corrections agree to FP32 rounding of the transfers (1e-6 of
the largest).  Levels smaller than a tile, ragged ones, either side of the size
limit, damped transfers, other numbers of steps on one side, W cycles (which
visit levels again), Galerkin operators, convection; with and without the
coarse cycle in one launch, bit-identical to each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("c1", dict(mx=1, my=1, mz=1, nref=3)), ("c1", dict(nref=4)), ("c1", dict(mx=3, my=2, mz=1, nref=5)),
         ("c1", dict(mx=5, my=2, mz=2, nref=5)), ("c1", dict(mx=2, my=3, mz=2, nref=4, nu1=1)),
         ("c1", dict(mx=2, my=3, mz=2, nref=4, nu2=3)),
         ("c1", dict(mx=3, my=2, mz=2, nref=4, damp_prol=0.8, damp_res=0.9)),
         ("c1", dict(mx=2, my=2, mz=3, nref=4, cycle=2)), ("c1", dict(mx=2, my=2, mz=3, nref=4, cycle=-1)),
         ("c1", dict(mx=2, my=2, mz=2, nref=4, rap=True)), ("c4", dict(mx=3, my=2, mz=2, nref=5)),
         ("c4", dict(mx=4, my=3, mz=2, nref=4))]


def _correction(name, over, fmt, coarse_levels):
    import ugcore_gb300 as ug
    from ugcore_gb300 import problems
    ctx = ug.Context(0)
    ctx.set_operator_format(fmt)
    ctx.set_tuning(coarse_levels=coarse_levels)
    p = problems.Problem(ctx, problems.config(name, precision="mixed", **over))
    d = ug.GPUVector(ctx, p.n).copy_from(np.random.default_rng(4).uniform(-1, 1, p.n))
    c = ug.GPUVector(ctx, p.n)
    p.gmg.apply(c, d)
    first = c.numpy()
    p.gmg.apply(c, d)
    assert np.array_equal(c.numpy(), first)
    return first


@pytest.mark.parametrize("name,over", CASES)
def test_matches_separate_steps(name, over):
    a, b = (_correction(name, over, "auto", levels) for levels in (0, -1))
    assert np.array_equal(a, b)
    ref = _correction(name, over, "sell", 0)
    assert np.abs(a - ref).max() <= 1e-6 * np.abs(ref).max()
