"""Gauss-Seidel on long, narrow grids and on large FP64 levels: a level whose few
lines of more than three rounds of a block would leave the GPU idle is swept colour
by colour, so is an FP64 level of 27 diagonals above 700000 rows, any other line by
line; the same corrections as the SELL format's, to rounding of the
transfers (1e-13 of the largest entry in FP64, 1e-6 in FP32)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _correction(fmt, elem, m, nref, precision):
    import ugcore_gb300 as ug
    ctx = ug.Context(0)
    ctx.set_operator_format(fmt)
    hier = ug.StructuredHierarchy(ctx, elem, *m, nref)
    disc = ug.DomainDiscretization(hier)
    rng = np.random.default_rng(2)
    disc.set_log_diffusion(rng.normal(size=hier.num_elements()))
    disc.set_source(rng.uniform(-1, 1, hier.num_vertices()))
    A, b = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, hier.num_vertices())
    disc.assemble_linear(A, b)
    g = ug.GeometricMultiGrid(disc)
    g.set_smoother(ug.GaussSeidel(1.0))
    g.set_precision(precision)
    g.init(A)
    c = ug.GPUVector(ctx, b.n)
    g.apply(c, b)
    out = c.numpy()
    ctx.profile_begin()
    g.apply(c, b)
    prof = ctx.profile_end()
    assert np.array_equal(c.numpy(), out)
    return out, any(k.startswith("L%d|" % nref) and "k_mcgs_lines" in k for k in prof)


# vertices per line 1505, 1537 (three and four rounds of 256 threads per colour),
# few lines of them; 1537 with 80 and with 144 lines per set; 3D
@pytest.mark.parametrize("elem,m,nref,lines", [("quad", (47, 1, 1), 5, True), ("quad", (48, 1, 1), 5, False),
                                               ("quad", (48, 5, 1), 5, False),
                                               ("quad", (48, 9, 1), 5, True), ("hex", (192, 1, 1), 3, False),
                                               ("tet", (256, 2, 1), 3, False)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 1e-6)])
def test_route_and_result(elem, m, nref, lines, precision, tol):
    got, used = _correction("auto", elem, m, nref, precision)
    assert used == lines
    want, _ = _correction("sell", elem, m, nref, precision)
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("precision,tol,lines", [("fp64", 1e-13, False), ("mixed", 1e-6, True)])
def test_one_block_of_two_rounds(precision, tol, lines):
    """513 x 3 x 3: one block per set, bound by one SM's FP64 pipe in FP64"""
    got, used = _correction("auto", "hex", (256, 1, 1), 1, precision)
    assert used == lines
    want, _ = _correction("sell", "hex", (256, 1, 1), 1, precision)
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("m,precision,tol,lines", [((5, 5, 5), "fp64", 1e-13, True), ((6, 5, 6), "fp64", 1e-13, False),
                                                   ((6, 5, 6), "mixed", 1e-6, True)])
def test_large_fp64_levels(m, precision, tol, lines):
    """81^3 and 97 x 81 x 97 hexahedra: 531441 and 762129 rows"""
    got, used = _correction("auto", "hex", m, 4, precision)
    assert used == lines
    want, _ = _correction("sell", "hex", m, 4, precision)
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
