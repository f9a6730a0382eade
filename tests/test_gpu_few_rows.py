"""Products of few rows of unstructured levels (SELL, whole rows loaded ahead of
the launch wait, as many slots as the rows are wide: triangles 7 entries,
quadrilaterals 9, tetrahedra 15 to 24, hexahedra 27, fans of up to 28) against a
two-level cycle in numpy from the exported operators and transfers.  A row sums
at most 28 products in two steps, a transfer and a base solve: 1e-12 of the
largest correction in FP64, 1e-5 in FP32 (6e-8 per operation)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(kind):
    if kind == "fan":       # 27 triangles around each of two vertices
        x, e = [], []
        for q in range(2):
            t = np.linspace(0, 2 * np.pi, 28)[:-1]
            n = len(x)
            x += [[3.0 * q, 0.0]] + [[3.0 * q + np.cos(s), np.sin(s)] for s in t]
            e += [[n, n + 1 + i, n + 1 + (i + 1) % 27] for i in range(27)]
        return "tri", np.array(x), np.array(e)
    m = {"tri": 9, "quad": 9, "tet": 4, "hex": 5}[kind]
    g = np.arange(m + 1)
    if kind in ("tri", "quad"):
        x = np.array([[i, j] for j in g for i in g], float)
        a = np.array([i + (m + 1) * j for j in range(m) for i in range(m)])
        q = np.stack([a, a + 1, a + m + 2, a + m + 1], 1)
        return kind, x, q if kind == "quad" else np.vstack([q[:, [0, 1, 2]], q[:, [0, 2, 3]]])
    x = np.array([[i, j, k] for k in g for j in g for i in g], float)
    ny, nz = m + 1, (m + 1) ** 2
    a = np.array([i + ny * j + nz * k for k in range(m) for j in range(m) for i in range(m)])
    c = np.stack([a, a + 1, a + 1 + ny, a + ny, a + nz, a + 1 + nz, a + 1 + ny + nz, a + ny + nz], 1)
    if kind == "hex":
        return kind, x, c
    return kind, x, np.vstack([c[:, p] for p in ([0, 1, 2, 6], [0, 1, 5, 6], [0, 3, 2, 6], [0, 3, 7, 6], [0, 4, 5, 6],
                                                [0, 4, 7, 6])])


def _csr(t, shape):
    import scipy.sparse as sp
    return sp.csr_matrix((t[2], t[1], t[0]), shape=shape)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("kind", ["tri", "quad", "tet", "hex", "fan"])
def test_two_level_cycle(kind, precision, tol):
    pytest.importorskip("scipy")
    import ugcore_gb300 as ug
    elem, x, e = _mesh(kind)
    ctx = ug.Context(0)
    hier = ug.UnstructuredHierarchy.from_arrays(ctx, elem, x, e, num_refinements=1)
    disc = ug.DomainDiscretization(hier)
    rng = np.random.default_rng(1)
    disc.set_log_diffusion(rng.normal(size=hier.num_elements()))
    disc.set_source_uniform(1)
    A, b = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, hier.num_vertices())
    disc.assemble_linear(A, b)
    g = ug.GeometricMultiGrid(disc)
    g.set_smoother(ug.Jacobi(0.6))
    g.set_precision(precision)
    g.init(A)
    d = rng.uniform(-1, 1, b.n)
    c = ug.GPUVector(ctx, b.n)
    g.apply(c, ug.GPUVector(ctx, b.n).copy_from(d))
    n0 = hier.num_vertices(0)
    A1, A0 = _csr(g.level_matrix(1), (b.n, b.n)), _csr(g.level_matrix(0), (n0, n0)).toarray()
    P, R = _csr(g.transfer(1, 0), (b.n, n0)), _csr(g.transfer(1, 1), (n0, b.n))
    w, want = 0.6 / A1.diagonal(), np.zeros(b.n)

    def smooth(d, want):
        for _ in range(2):
            s = w * d
            want += s
            d = d - A1 @ s
        return d

    d = smooth(d, want)
    t = P @ np.linalg.solve(A0, R @ d)
    want += t
    smooth(d - A1 @ t, want)
    assert np.abs(c.numpy() - want).max() <= tol * np.abs(want).max()
