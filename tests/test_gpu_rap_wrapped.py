"""Galerkin levels of a top operator that couples vertices across the grid: the
rows of R and P at boundary vertices (weight 1 at a coinciding vertex) carry
such an entry down, where it falls on an offset of the element stencil, so the
kernels that take a neighbour outside the grid as absent (2D and small 3D levels
in two launches, Gauss-Seidel by lines) must leave these levels to the others.
Against the SELL format, which keeps every entry's column: 1e-12 of the largest
correction in FP64, 1e-6 in FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OUTSIDE_IS_ABSENT = ("k_pre2d", "k_post2d", "k_pre3d", "k_post3d", "k_mcgs_lines")


def _wrapped(ug, A, nx, ny, nz, dy):
    """A with entries (nx-1, j, k) -> (0, j + dy, k) of -0.01 at even j, k"""
    import scipy.sparse as sp
    rp, ci, va = A.export_csr()
    n = len(rp) - 1
    k, j = np.meshgrid(np.arange(0, nz, 2), np.arange(0, ny - dy, 2), indexing="ij")
    row = (nx - 1 + nx * (j + ny * k)).ravel()
    W = sp.csr_matrix((np.full(len(row), -0.01), (row, row + 1 - nx + dy * nx)), shape=(n, n))
    S = (sp.csr_matrix((va, ci, rp), shape=(n, n)) + W).tocsr()
    S.sort_indices()
    return ug.GPUSparseMatrix(A.ctx).set_csr(S.indptr, S.indices, S.data)


def _multigrid(fmt, name, over, dy, profile=False):
    import ugcore_gb300 as ug
    from ugcore_gb300 import problems
    ctx = ug.Context(0)
    ctx.set_operator_format(fmt)
    cfg = problems.config(name, rap=True, **over)
    p = problems.Problem(ctx, cfg)
    f = 2 ** cfg["nref"]
    nx, ny, nz = cfg["mx"] * f + 1, cfg["my"] * f + 1, (cfg["mz"] * f + 1 if p.hier.dim == 3 else 1)
    g = p._make_gmg(transposed=False)
    g.init(_wrapped(ug, p.A, nx, ny, nz, dy))
    # the entry is there on the level below the top
    l = p.hier.num_levels - 2
    rp, ci, va = g.level_matrix(l)
    cnx = (nx + 1) // 2
    e = slice(rp[cnx - 1], rp[cnx])
    assert np.any(np.isclose(va[e][ci[e] == (dy // 2) * cnx], -0.01))
    d = ug.GPUVector(ctx, p.n).copy_from(np.random.default_rng(4).uniform(-1, 1, p.n))
    c = ug.GPUVector(ctx, p.n)
    if profile:
        ctx.profile_begin()
    g.apply(c, d)
    return c.numpy(), (ctx.profile_end() if profile else None)


@pytest.mark.parametrize("name,over,tol", [
    ("c3", dict(mx=2, my=2, nref=4, precision="fp64"), 1e-12),
    ("c3", dict(mx=3, my=2, nref=5, precision="mixed"), 1e-6),
    ("c1", dict(mx=2, my=2, mz=2, nref=3, precision="mixed"), 1e-6),
    ("c1", dict(mx=3, my=2, mz=2, nref=4, precision="mixed"), 1e-6)])
def test_jacobi_keeps_the_coupling(name, over, tol):
    got, want = (_multigrid(f, name, over, 0)[0] for f in ("auto", "sell"))
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("smoother", ["mcgs", "mcbgs", "mcsgs"])
@pytest.mark.parametrize("name,over", [("c3", dict(mx=2, my=2, nref=4)), ("c1", dict(mx=2, my=2, mz=2, nref=3))])
def test_no_kernel_that_drops_it(name, over, smoother):
    """offset 1 on the lower levels: vertices of two colours, and (on the top
    level) two of one colour, whose order is open: only the kernels are compared"""
    prof = _multigrid("auto", name, dict(over, smoother=smoother), 2, profile=True)[1]
    assert not [k for k in prof if any(q in k for q in OUTSIDE_IS_ABSENT)]
