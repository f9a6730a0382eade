"""Gauss-Seidel sweeps of structured levels line by line (k_mcgs_lines) against
the colour-by-colour kernels that the SELL format keeps: the same operations in
the same order, so multigrid corrections agree to rounding of the transfers
(1e-13 of the largest entry in FP64; the FP32 sums are the same to 1e-6).
Odd and even counts of lines, lines of more than 512 vertices, 2D and 3D, the
three kinds with and without relaxation, a top operator that couples vertices
across the ends of grid lines."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [("quad", (2, 3, 1), 3), ("quad", (5, 2, 1), 7), ("hex", (2, 3, 2), 2), ("hex", (3, 2, 2), 3),
         ("tet", (2, 2, 3), 2), ("tet", (5, 3, 2), 1)]


def _correction(ug, fmt, elem, m, nref, kind, relax, precision, wrap=False):
    ctx = ug.Context(0)
    ctx.set_operator_format(fmt)
    hier = ug.StructuredHierarchy(ctx, elem, *m, nref)
    disc = ug.DomainDiscretization(hier)
    rng = np.random.default_rng(2)
    disc.set_log_diffusion(rng.normal(size=hier.num_elements()))
    disc.set_source(rng.uniform(-1, 1, hier.num_vertices()))
    A, b = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, hier.num_vertices())
    disc.assemble_linear(A, b)
    if wrap:
        # couple each line's last inner vertex with the next line's first one
        import scipy.sparse as sp
        rp, ci, va = A.export_csr()
        S = sp.csr_matrix((va, ci, rp)).tolil()
        nx = m[0] * 2 ** nref + 1
        for r in range(2 * nx - 1, b.n - nx, nx):
            S[r, r + 1] = S[r + 1, r] = -0.01
        S = S.tocsr()
        S.sort_indices()
        A.set_csr(S.indptr, S.indices, S.data)
    g = ug.GeometricMultiGrid(disc)
    g.set_smoother(kind(relax))
    g.set_precision(precision)
    g.init(A)
    d = ug.GPUVector(ctx, b.n).copy_from(rng.uniform(-1, 1, b.n))
    c = ug.GPUVector(ctx, b.n)
    g.apply(c, d)
    first = c.numpy()
    g.apply(c, d)
    assert np.array_equal(c.numpy(), first)
    return first


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 1e-6)])
@pytest.mark.parametrize("kind,relax", [("GaussSeidel", 1.0), ("BackwardGaussSeidel", 0.8),
                                        ("SymmetricGaussSeidel", 1.1)])
@pytest.mark.parametrize("elem,m,nref", GRIDS)
def test_lines_match_colours(elem, m, nref, kind, relax, precision, tol):
    import ugcore_gb300 as ug
    got, want = (_correction(ug, f, elem, m, nref, getattr(ug, kind), relax, precision) for f in ("auto", "sell"))
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("elem,m,nref", [GRIDS[0], GRIDS[2]])
def test_couplings_across_line_ends(elem, m, nref):
    pytest.importorskip("scipy")
    import ugcore_gb300 as ug
    got, want = (_correction(ug, f, elem, m, nref, ug.GaussSeidel, 1.0, "fp64", wrap=True) for f in ("auto", "sell"))
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
