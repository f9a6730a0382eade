"""Diagonal layout without its all-zero diagonals (op_from_csr): products and
multigrid corrections where the left-out entries stay zero, become nonzero in a
refill of the same pattern, or stand in rows whose columns are not sorted.

Reference: the product in numpy from the matrix's own CRS arrays; each row sums
at most 27 products, so 27 rounding errors of its largest partial sum bound the
difference (1e-14 times the row's sum of |a_ij x_j|).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check_product(ug, ctx, A, seed=1):
    rp, ci, va = A.export_csr()
    n = len(rp) - 1
    x = np.random.default_rng(seed).uniform(-1, 1, n)
    rows = np.repeat(np.arange(n), np.diff(rp))
    want = np.bincount(rows, va * x[ci], n)
    scale = np.bincount(rows, np.abs(va * x[ci]), n)
    xv, yv = ug.GPUVector(ctx, n).copy_from(x), ug.GPUVector(ctx, n)
    A.apply(yv, xv)
    assert np.all(np.abs(yv.numpy() - want) <= 1e-14 * scale)


@pytest.mark.parametrize("elem,m,nref", [("tet", (2, 2, 2), 1), ("tet", (5, 3, 2), 2), ("tet", (4, 4, 4), 3),
                                         ("hex", (2, 3, 2), 2), ("quad", (3, 5, 1), 3)])
def test_products_before_and_after_entries_become_nonzero(elem, m, nref):
    import ugcore_gb300 as ug
    ctx = ug.Context(0)
    hier = ug.StructuredHierarchy(ctx, elem, *m, nref)
    disc = ug.DomainDiscretization(hier)
    disc.set_source_uniform(3)
    A, b = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, hier.num_vertices())
    disc.assemble_linear(A, b)
    _check_product(ug, ctx, A)
    rp, ci, va = A.export_csr()
    zero = np.flatnonzero(va == 0.0)
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    pick = zero[:: max(1, len(zero) // 7)]
    A.add_entries(rows[pick], ci[pick], np.linspace(0.5, 1.5, len(pick)))
    _check_product(ug, ctx, A)
    # the assembled values again, then with every entry 0, then one diagonal only
    disc.assemble_linear(A, b)
    _check_product(ug, ctx, A)
    A.clear_retain_structure()
    _check_product(ug, ctx, A)
    diag = np.flatnonzero(rows == ci)
    A.add_entries(rows[diag], ci[diag], np.arange(1.0, len(diag) + 1))
    _check_product(ug, ctx, A)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
def test_rows_in_any_column_order(n):
    import ugcore_gb300 as ug
    ctx = ug.Context(0)
    rng = np.random.default_rng(n)
    offs = [o for o in (-37, -5, -1, 0, 1, 5, 37) if abs(o) < n]
    rp, ci = [0], []
    for r in range(n):
        c = [r + o for o in offs if 0 <= r + o < n]
        ci += list(rng.permutation(c))
        rp.append(len(ci))
    va = rng.uniform(-1, 1, len(ci))
    va[np.array(ci) - np.repeat(np.arange(n), np.diff(rp)) == 5] = 0.0
    A = ug.GPUSparseMatrix(ctx).set_csr(rp, ci, va)
    _check_product(ug, ctx, A)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_multigrid_follows_entries_that_become_nonzero(precision):
    import ugcore_gb300 as ug
    ctx = ug.Context(0)
    hier = ug.StructuredHierarchy(ctx, "tet", 3, 2, 2, 2)
    disc = ug.DomainDiscretization(hier)
    disc.set_source_uniform(3)
    A, b = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, hier.num_vertices())
    disc.assemble_linear(A, b)

    def correction(g):
        c = ug.GPUVector(ctx, b.n)
        g.apply(c, b)
        return c.numpy()

    def multigrid():
        g = ug.GeometricMultiGrid(disc)
        g.set_precision(precision)
        return g

    g = multigrid()
    g.init(A)
    first = correction(g)
    rp, ci, va = A.export_csr()
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    zero = np.flatnonzero((va == 0.0) & (rows != ci))
    A.add_entries(rows[zero], ci[zero], np.full(len(zero), 0.01))
    g.init(A)
    fresh = multigrid()
    fresh.init(A)
    got = correction(g)
    assert np.array_equal(got, correction(fresh))
    assert not np.array_equal(got, first)
    # back to the assembled operator: the first correction, bit for bit
    disc.assemble_linear(A, b)
    g.init(A)
    assert np.array_equal(correction(g), first)
