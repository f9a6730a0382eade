"""State that calls share: BiCGStab's FP32 copies of its search direction and
half-step defect across restarts, and the one flag of a context that reports
values at left-out diagonals, with several operators and multigrids beside each
other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("restart", [2, 4, 6])
def test_restarts_with_a_mixed_precision_multigrid(restart):
    """the defects of the first half steps, with restarts among them, follow
    those of the FP64 multigrid: its correction is perturbed by some 1e-6
    (FP32), each half step's factors with it: 1e-3 leaves room for eight of
    them, a correction of another vector changes the defect by its own size"""
    import ugcore_gb300 as ug
    from ugcore_gb300 import problems
    ctx = ug.Context(0)
    out = []
    for precision in ("fp64", "mixed"):
        p = problems.Problem(ctx, problems.config("c4", nref=3, precision=precision, bicg_restart=restart))
        st = p.solve()
        assert st["converged"]
        r = ug.GPUVector(ctx, p.n)
        p.A.apply(r, p.x)
        assert np.linalg.norm(r.numpy() - p.b.numpy()) <= 1e-9 * np.linalg.norm(p.b.numpy())
        out.append(np.array(p.solver.history())[:9])
    assert np.all(np.abs(out[1] - out[0]) <= 1e-3 * out[0])


def _case(ug, ctx, seed):
    """a Kuhn-tetrahedral operator and its multigrid, set up and used once"""
    hier = ug.StructuredHierarchy(ctx, "tet", 2, 2, 2 + seed, 2)
    disc = ug.DomainDiscretization(hier)
    disc.set_source_uniform(seed)
    disc.set_log_diffusion(np.random.default_rng(seed).normal(size=hier.num_elements()))
    A, b = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, hier.num_vertices())
    g = ug.GeometricMultiGrid(disc)
    g.set_precision("mixed" if seed % 2 else "fp64")

    def prepare(extra):
        disc.assemble_linear(A, b)
        if extra:
            rp, ci, va = A.export_csr()
            rows = np.repeat(np.arange(b.n), np.diff(rp))
            zero = np.flatnonzero((va == 0.0) & (rows != ci))[::5]
            A.add_entries(rows[zero], ci[zero], np.full(len(zero), 0.01))

    def results():
        c = ug.GPUVector(ctx, b.n)
        g.apply(c, b)
        y = ug.GPUVector(ctx, b.n)
        A.apply(y, c)
        return c.numpy(), y.numpy()

    prepare(False)
    g.init(A)
    results()
    return prepare, lambda: g.init(A), results


@pytest.mark.parametrize("order", ["extra first", "extra last", "both"])
def test_multigrids_with_and_without_left_out_diagonals(order):
    """three multigrids in one context, their operators changed, and then all set
    up again before any is used, against a context of its own for each"""
    import ugcore_gb300 as ug
    extra = {"extra first": (True, False, False), "extra last": (False, False, True), "both": (True, False, True)}[order]
    ctx = ug.Context(0)
    cases = [_case(ug, ctx, s) for s in range(3)]
    for (prepare, _, _), x in zip(cases, extra):
        prepare(x)
    for _, init, _ in cases:
        init()
    got = [results() for _, _, results in cases]
    for s in range(3):
        prepare, init, results = _case(ug, ug.Context(0), s)
        prepare(extra[s])
        init()
        for a, b in zip(got[s], results()):
            assert np.array_equal(a, b)
