"""The coarse cycle where levels are prepared for two Jacobi steps per pass
(sweep_fusion): it takes the smallest of them, the larger ones keep their fused
launches, and corrections are bit-identical to separate launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,over,taken,left", [("c2", dict(mx=1, my=4, mz=1, nref=4), 2, 3),
                                                  ("c1", dict(nref=4), 1, 2)])
def test_smallest_levels_join(name, over, taken, left):
    """taken, left: the finest level in the coarse cycle, the next one"""
    import ugcore_gb300 as ug
    from ugcore_gb300 import problems
    out = []
    for tuning in (dict(coarse_levels=-1, sweep_fusion=3), dict(coarse_levels=0, sweep_fusion=3)):
        ctx = ug.Context(0)
        ctx.set_tuning(**tuning)
        p = problems.Problem(ctx, problems.config(name, precision="mixed", **over))
        d = ug.GPUVector(ctx, p.n).copy_from(np.random.default_rng(3).uniform(-1.0, 1.0, p.n))
        c = ug.GPUVector(ctx, p.n)
        p.gmg.apply(c, d)
        out.append(c.numpy())
        ctx.profile_begin()
        p.gmg.apply(c, d)
        prof = ctx.profile_end()
        fused = {int(k[1:k.index("|")]) for k in prof if "k_sweep2" in k}
        coarse = [k for k in prof if "k_coarse_cycle" in k]
        if tuning["coarse_levels"] < 0:
            assert len(coarse) == 1 and coarse[0].startswith("L0-%d|" % taken)
            assert left in fused and taken not in fused
        else:
            assert not coarse
    assert np.array_equal(out[0], out[1])
