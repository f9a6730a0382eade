"""Re-initialisation of Kuhn-tetrahedral levels queues its work without a wait:
their diagonal layouts leave out the entries that the assembly writes as exact
zeros, and nothing is read back to test them.  A kernel that keeps the stream
busy for some 0.2 s is queued first; the calls must return before it ends.  Where
values come from elsewhere the entries are tested, and a layout that lacks one
is rebuilt."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _set_up(precision, transposed=False, const=False):
    import ugcore_gb300 as ug
    ctx = ug.Context(0)
    hier = ug.StructuredHierarchy(ctx, "tet", 2, 3, 2, 3)
    disc = ug.DomainDiscretization(hier)
    disc.set_source_uniform(3)
    if not const:
        disc.set_log_diffusion(np.random.default_rng(1).normal(size=hier.num_elements()))
    A, b = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, hier.num_vertices())
    g = ug.GeometricMultiGrid(disc)
    g.set_precision(precision)
    g.set_transposed(transposed)
    s = ug.CG(ctx)
    s.set_preconditioner(g)
    s.set_convergence_check(ug.StdConvCheck(50, 1e-300, 1e-9))
    return ug, ctx, hier, disc, A, b, g, s


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("transposed,const", [(False, False), (True, False), (False, True)])
def test_returns_before_the_stream_is_idle(precision, transposed, const):
    torch = pytest.importorskip("torch")
    ug, ctx, hier, disc, A, b, g, s = _set_up(precision, transposed, const)
    x, AT = ug.GPUVector(ctx, b.n), ug.GPUSparseMatrix(ctx)
    stream = torch.cuda.ExternalStream(ctx.stream)
    for busy in (False, False, True):
        disc.assemble_linear(A, b)
        if transposed:
            disc.adjoint_operator(A, AT)
        done = torch.cuda.Event()
        if busy:
            with torch.cuda.stream(stream):
                torch.cuda._sleep(400_000_000)
        done.record(stream)
        g.init(A)
        s.init(AT if transposed else A)
        if busy:
            assert not done.query()
        x.set(0.0)
        assert s.apply(x, b)
    rp, ci, va = (AT if transposed else A).export_csr()
    rows = np.repeat(np.arange(b.n), np.diff(rp))
    r = b.numpy() - np.bincount(rows, va * x.numpy()[ci], b.n)
    assert np.linalg.norm(r) <= 1e-8 * np.linalg.norm(b.numpy())


@pytest.mark.parametrize("change", ["entries", "copy", "velocity"])
def test_other_values_are_tested(change):
    """the operator after its zeros got values, by each kind of call that writes some"""
    ug, ctx, hier, disc, A, b, g, s = _set_up("fp64")
    disc.assemble_linear(A, b)
    x, y = ug.GPUVector(ctx, b.n), ug.GPUVector(ctx, b.n)
    x.copy_from(np.random.default_rng(4).uniform(-1, 1, b.n))
    A.apply(y, x)               # the layout without the zeros
    rp, ci, va = A.export_csr()
    rows = np.repeat(np.arange(b.n), np.diff(rp))
    zero = np.flatnonzero((va == 0.0) & (rows != ci))[::11]
    if change == "entries":
        A.add_entries(rows[zero], ci[zero], np.full(len(zero), 0.25))
    elif change == "copy":
        B = ug.GPUSparseMatrix(ctx)
        B.set_as_copy_of(A, 1.0)
        B.add_entries(rows[zero], ci[zero], np.full(len(zero), 0.25))
        A.set_as_copy_of(B, 2.0)
    else:
        class V:
            nmodes, scale = 1, 0.5
            k = np.array([[6.3, 1.0, 2.1]])
            phase = np.array([0.3])
            c = np.cross(k, np.array([[0.2, 1.0, -0.4]]))
        disc.set_velocity_field(V, 2.0)
        disc.set_upwind("full")
        disc.assemble_linear(A, b)
    A.apply(y, x)
    va = A.export_csr()[2]
    assert np.any(va[np.flatnonzero((np.abs(ci - rows) > 1) & (va != 0.0))])
    want = np.bincount(rows, va * x.numpy()[ci], b.n)
    scale = np.bincount(rows, np.abs(va * x.numpy()[ci]), b.n)
    assert np.all(np.abs(y.numpy() - want) <= 1e-14 * scale)
    # the assembled operator again: still with every entry at hand
    if change != "velocity":
        disc.assemble_linear(A, b)
        A.apply(y, x)
        va = A.export_csr()[2]
        want = np.bincount(rows, va * x.numpy()[ci], b.n)
        scale = np.bincount(rows, np.abs(va * x.numpy()[ci]), b.n)
        assert np.all(np.abs(y.numpy() - want) <= 1e-14 * scale)
