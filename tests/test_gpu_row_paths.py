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
