"""The kernels that take whole 2D levels, small 3D levels and Gauss-Seidel lines
against the separate kernels on the same diagonal layouts: the same bits.  The
operator set from arrays (a pattern of its own) with Galerkin levels keeps all
levels to the separate kernels, the assembled one with the same values takes the
others.  (FP64 2D levels of up to a block of rows per SM: above, the separate
kernels sum a row in one chain.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FUSED = ("k_pre2d", "k_post2d", "k_pre3d", "k_post3d", "k_mcgs_lines")


@pytest.mark.parametrize("name,over", [
    ("c3", dict(mx=3, my=2, nref=4, precision="fp64")), ("c3", dict(mx=2, my=2, nref=6, precision="fp64")),
    ("c3", dict(mx=3, my=2, nref=4, precision="mixed")), ("c3", dict(mx=2, my=3, nref=8, precision="mixed")),
    ("c1", dict(mx=2, my=3, mz=2, nref=4, precision="mixed")), ("c4", dict(mx=3, my=2, mz=2, nref=4)),
    ("c3", dict(mx=2, my=2, nref=6, precision="mixed", smoother="mcgs", damp=1.0)),
    ("c1", dict(mx=2, my=3, mz=2, nref=3, precision="fp64", smoother="mcsgs", damp=0.9)),
    ("c2", dict(mx=2, my=3, mz=2, nref=3, smoother="mcbgs", damp=1.0))])
def test_same_bits(name, over):
    import ugcore_gb300 as ug
    from ugcore_gb300 import problems
    ctx = ug.Context(0)
    p = problems.Problem(ctx, problems.config(name, rap=True, **over))
    B = ug.GPUSparseMatrix(ctx).set_csr(*p.A.export_csr())
    d = ug.GPUVector(ctx, p.n).copy_from(np.random.default_rng(4).uniform(-1, 1, p.n))
    out = []
    for A in (p.A, B):
        g = p._make_gmg(transposed=False)
        g.init(A)
        c = ug.GPUVector(ctx, p.n)
        g.apply(c, d)
        out.append(c.numpy())
        ctx.profile_begin()
        g.apply(c, d)
        prof = ctx.profile_end()
        assert any(q in k for k in prof for q in FUSED) == (A is p.A)
    assert np.array_equal(out[0], out[1])
