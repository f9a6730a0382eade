"""Structured levels assembled from their class matrices (k_fv1_rows.cu)
against the element-by-element kernels (row_assembly off): the time-discrete
operator and right-hand side, the stationary and time-discrete defect, the
adjoint gradients, on the smallest levels with interior rows, unequal sides,
and levels on either side of the one-launch limit of 65536 rows.

A row sums at most 64 element entries (hexahedra) and 27 products, the
geometry of a cell agrees with its class to a few roundings: 1e-13 of the
largest sum of absolute terms bounds the difference.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("quad", (2, 3, 1), 0, False), ("quad", (3, 2, 1), 3, False), ("quad", (4, 5, 1), 6, False),
         ("hex", (2, 2, 2), 0, False), ("hex", (3, 2, 4), 2, True), ("hex", (3, 3, 2), 4, False),
         ("tet", (2, 2, 2), 0, False), ("tet", (2, 5, 3), 2, True), ("tet", (3, 2, 3), 4, False)]


class _Velocity:
    nmodes, scale = 2, 0.3
    k = np.array([[6.3, 0.0, 2.1], [-3.0, 5.0, 1.0]])
    phase = np.array([0.3, 1.7])
    c = np.cross(k, np.array([[0.2, 1.0, -0.4], [0.7, 0.1, 0.5]]))


def _all(ug, rows, elem, m, nref, flow, const, theta):
    ctx = ug.Context(0)
    ctx.set_tuning(row_assembly=rows)
    hier = ug.StructuredHierarchy(ctx, elem, *m, nref)
    disc = ug.DomainDiscretization(hier)
    n, ne = hier.num_vertices(), hier.num_elements()
    rng = np.random.default_rng(5)
    if const:
        disc.set_diffusion(0.7)
    else:
        disc.set_log_diffusion(rng.normal(size=ne))
    if flow:
        disc.set_velocity_field(_Velocity, 2.0)
        disc.set_upwind("full")
    disc.set_source(rng.uniform(-1, 1, n))
    u, u_old, lam = (ug.GPUVector(ctx, n).copy_from(rng.uniform(-1, 1, n)) for _ in range(3))
    A, b, d, dt = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, n), ug.GPUVector(ctx, n), ug.GPUVector(ctx, n)
    td = ug.ThetaTimeStep(disc, theta)
    td.prepare_step(u_old, 0.0, 0.05)
    td.assemble_linear(A, b)
    disc.assemble_defect(d, u)
    td.assemble_defect(dt, u)
    J = ug.GPUSparseMatrix(ctx)
    td.assemble_jacobian(J)
    S, sb = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, n)
    disc.assemble_linear(S, sb)
    return dict(A=A.export_csr(), b=b.numpy(), d=d.numpy(), dt=dt.numpy(), J=J.export_csr()[2],
                S=S.export_csr(), sb=sb.numpy(), gm=disc.grad_logk(u, lam), gf=disc.grad_source(lam),
                u=u.numpy(), u_old=u_old.numpy(), lam=lam.numpy())


@pytest.mark.parametrize("const,theta", [(False, 0.5), (True, 0.5), (True, 1.0)])
@pytest.mark.parametrize("elem,m,nref,flow", CASES)
def test_rows_match_elements(elem, m, nref, flow, const, theta):
    import ugcore_gb300 as ug
    got, want = (_all(ug, r, elem, m, nref, flow, const, theta) for r in (2, 0))
    for k in ("A", "S"):
        assert np.array_equal(got[k][0], want[k][0]) and np.array_equal(got[k][1], want[k][1])
        assert np.abs(got[k][2] - want[k][2]).max() <= 1e-13 * np.abs(want[k][2]).max()
    assert np.abs(got["J"] - want["J"]).max() <= 1e-13 * np.abs(want["J"]).max()
    rp, ci, va = want["S"]
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    # |A| |u| + |b| with every |u| at most 1; |V| <= |b| / |f| enters below it
    scale = np.bincount(rows, np.abs(va)).max() + np.abs(want["sb"]).max()
    tscale = scale + np.abs(want["A"][2]).max() + np.abs(want["b"]).max()
    assert np.abs(got["d"] - want["d"]).max() <= 1e-13 * scale
    assert np.abs(got["b"] - want["b"]).max() <= 1e-13 * tscale
    assert np.abs(got["dt"] - want["dt"]).max() <= 1e-13 * tscale
    assert np.abs(got["gm"] - want["gm"]).max() <= 1e-13 * scale * (27 if elem == "hex" else 8)
    assert np.abs(got["gf"] - want["gf"]).max() <= 1e-13 * np.abs(want["gf"]).max()


def _mesh(kind, seed=2):
    """a moved box of simplices, or a fan whose hub row is long"""
    rng = np.random.default_rng(seed)
    if kind == "fan":       # triangles around one vertex: a row of 81 entries
        t = np.linspace(0, 2 * np.pi, 81)[:-1]
        x = np.vstack([[0.0, 0.0], np.c_[np.cos(t), np.sin(t)]])
        return x, np.array([[0, 1 + i, 1 + (i + 1) % 80] for i in range(80)])
    if kind == "stack":     # tetrahedra around one edge, 20 rings of their own: rows of 62 entries
        x, e = [], []
        for q in range(20):
            t = np.linspace(0, 2 * np.pi, 61)[:-1]
            n = len(x)
            x += [[0.0, 0.0, 3.0 * q], [0.0, 0.0, 3.0 * q + 1]]
            x += [[np.cos(s), np.sin(s), 3.0 * q + 0.5] for s in t]
            e += [[n, n + 2 + i, n + 2 + (i + 1) % 60, n + 1] for i in range(60)]
        return np.array(x), np.array(e)
    if kind == "tri":
        m = 5
        x = np.array([[i, j] for j in range(m + 1) for i in range(m + 1)], float)
        inner = ((x > 0) & (x < m)).all(1)
        x[inner] += rng.uniform(-0.2, 0.2, (inner.sum(), 2))
        e = []
        for j in range(m):
            for i in range(m):
                a = i + (m + 1) * j
                e += [[a, a + 1, a + m + 2], [a, a + m + 2, a + m + 1]]
        return x, np.array(e)
    m = 2 if kind == "tet" else 3
    x = np.array([[i, j, k] for k in range(m + 1) for j in range(m + 1) for i in range(m + 1)], float)
    inner = ((x > 0) & (x < m)).all(1)
    x[inner] += rng.uniform(-0.2, 0.2, (inner.sum(), 3))
    e = []
    for k in range(m):
        for j in range(m):
            for i in range(m):
                for p in ((0, 1), (0, 2), (1, 0), (1, 2), (2, 0), (2, 1)):
                    c = np.array([[i, j, k]] * 4)
                    c[1:, p[0]] += 1
                    c[2:, p[1]] += 1
                    c[3:, 3 - p[0] - p[1]] += 1
                    q = c[:, 0] + (m + 1) * (c[:, 1] + (m + 1) * c[:, 2])
                    e.append(q if np.linalg.det(x[q[1:]] - x[q[0]]) > 0 else q[[0, 2, 1, 3]])
    return x, np.array(e)


@pytest.mark.parametrize("theta", [0.5, 1.0])
@pytest.mark.parametrize("kind,nref", [("tri", 0), ("tri", 4), ("fan", 0), ("stack", 0), ("tet", 0), ("tet", 1), ("tet", 3),
                                       ("tet3", 2)])
def test_gathered_rows_match_elements(kind, nref, theta):
    """unstructured simplices (k_fv1_gather.cu) against the element kernel:
    operator and right-hand side, stationary and time-discrete, with Dirichlet
    vertices all around and with one Dirichlet vertex only, short and long rows"""
    import ugcore_gb300 as ug
    x, e = _mesh(kind)
    one = np.zeros(len(x), np.uint8)
    one[0] = 1
    for dirichlet in (None, one):
        got = []
        for rows in (2, 0):
            ctx = ug.Context(0)
            ctx.set_tuning(row_assembly=rows)
            hier = ug.UnstructuredHierarchy.from_arrays(ctx, "tet" if x.shape[1] == 3 else "tri", x, e,
                                                        dirichlet_vertices=dirichlet, num_refinements=nref)
            disc = ug.DomainDiscretization(hier)
            n = hier.num_vertices()
            rng = np.random.default_rng(5)
            disc.set_log_diffusion(rng.normal(size=hier.num_elements()))
            disc.set_source(rng.uniform(-1, 1, n))
            u_old = ug.GPUVector(ctx, n).copy_from(rng.uniform(-1, 1, n))
            A, b = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, n)
            td = ug.ThetaTimeStep(disc, theta)
            td.prepare_step(u_old, 0.0, 0.05)
            for _ in range(2):      # fresh and kept pattern
                disc.assemble_linear(A, b)
                s = A.export_csr() + (b.numpy(),)
                td.assemble_linear(A, b)
            got.append(s + A.export_csr()[2:] + (b.numpy(),))
        (rp, ci, va, b0, vt, b1), want = got
        assert np.array_equal(rp, want[0]) and np.array_equal(ci, want[1])
        # an entry sums the elements around an edge, each from a few products
        # of edge vectors: 1e-12 of the row's largest entry leaves room for
        # their cancellation on moved meshes
        for v, w in ((va, want[2]), (vt, want[4])):
            row_max = np.maximum.reduceat(np.abs(w), rp[:-1])
            assert np.all(np.abs(v - w) <= 1e-12 * np.repeat(row_max, np.diff(rp)))
        rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
        scale = np.bincount(rows, np.abs(want[2])).max() + np.abs(want[3]).max()
        assert np.abs(b0 - want[3]).max() <= 1e-13 * np.abs(want[3]).max()
        assert np.abs(b1 - want[5]).max() <= 1e-12 * (scale + np.abs(want[5]).max())
