"""2D levels in two launches (k_level2d.cu) against the step-by-step kernels of
the SELL format: the same row operations; an FP64 row may be summed in two
chains (1e-12 of the largest correction), FP32 ones are the same to 1e-6.
Levels smaller than a tile, ragged ones, either side of the size limit, damped
transfers, other numbers of steps on one side, W cycles (which visit levels
again), Galerkin operators, solves with the fused (z, r)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(dict(mx=1, my=1, nref=2), {}), (dict(mx=2, my=2, nref=3), {}), (dict(mx=5, my=3, nref=4), {}),
         (dict(mx=2, my=7, nref=5), dict(nu1=1)), (dict(mx=2, my=7, nref=5), dict(nu2=3)),
         (dict(mx=3, my=2, nref=5), dict(damp_prol=0.8, damp_res=0.9)), (dict(mx=2, my=2, nref=5), dict(cycle=2)),
         (dict(mx=2, my=2, nref=5), dict(cycle=-1)), (dict(mx=2, my=2, nref=5), dict(rap=True)),
         (dict(mx=2, my=2, nref=7), {}), (dict(mx=5, my=5, nref=6), {}), (dict(mx=4, my=5, nref=7), {})]


def _problem(fmt, grid, over, precision):
    import ugcore_gb300 as ug
    from ugcore_gb300 import problems
    ctx = ug.Context(0)
    ctx.set_operator_format(fmt)
    return problems.Problem(ctx, problems.config("c3", precision=precision, **grid, **over))


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-6)])
@pytest.mark.parametrize("grid,over", CASES)
def test_matches_separate_steps(grid, over, precision, tol):
    import ugcore_gb300 as ug
    out = []
    for fmt in ("auto", "sell"):
        p = _problem(fmt, grid, over, precision)
        d = ug.GPUVector(p.ctx, p.n).copy_from(np.random.default_rng(4).uniform(-1, 1, p.n))
        c = ug.GPUVector(p.ctx, p.n)
        p.gmg.apply(c, d)
        first = c.numpy()
        p.gmg.apply(c, d)
        assert np.array_equal(c.numpy(), first)
        out.append(first)
    assert np.abs(out[0] - out[1]).max() <= tol * np.abs(out[1]).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grid", [dict(mx=2, my=2, nref=6), dict(mx=3, my=4, nref=5)])
def test_solves_take_the_same_steps(grid, precision):
    a, b = (_problem(fmt, grid, {}, precision) for fmt in ("auto", "sell"))
    sa, sb = a.solve(), b.solve()
    assert sa["ok"] and sb["ok"] and abs(sa["steps"] - sb["steps"]) <= 1
    # both residuals are below 1e-10 of |b|: the solutions agree to some 1e-8
    assert np.abs(a.x.numpy() - b.x.numpy()).max() <= 1e-8 * np.abs(b.x.numpy()).max()
