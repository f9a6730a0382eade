"""Memory of the row-wise assembly of unstructured simplex levels
(k_fv1_gather.cu): one workspace for all levels, and the element kernels where
the device has no memory left for it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _kuhn(m):
    e, g = [], np.arange(m + 1)
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:, ::-1].astype(float)
    for k in range(m):
        for j in range(m):
            for i in range(m):
                for p in ((0, 1), (0, 2), (1, 0), (1, 2), (2, 0), (2, 1)):
                    c = np.array([[i, j, k]] * 4)
                    c[1:, p[0]] += 1
                    c[2:, p[1]] += 1
                    c[3:, 3 - p[0] - p[1]] += 1
                    e.append(c[:, 0] + (m + 1) * (c[:, 1] + (m + 1) * c[:, 2]))
    return x, np.array(e)


def _disc(ug, nref, m=3):
    ctx = ug.Context(0)
    x, e = _kuhn(m)
    hier = ug.UnstructuredHierarchy.from_arrays(ctx, "tet", x, e, num_refinements=nref)
    disc = ug.DomainDiscretization(hier)
    disc.set_source_uniform(3)
    return ctx, hier, disc


def _memory_of_operators(rows):
    """device memory that assembling every level takes, and the levels' sizes;
    all of it is given back on return"""
    torch = pytest.importorskip("torch")
    import ugcore_gb300 as ug
    ctx, hier, disc = _disc(ug, 5)
    ctx.set_tuning(row_assembly=rows)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    keep = []
    for l in range(hier.num_levels - 1, -1, -1):
        A = ug.GPUSparseMatrix(ctx)
        disc.assemble_jacobian(A, l)
        keep.append(A)
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    return used, [(hier.num_vertices(l), hier.num_elements(l)) for l in range(hier.num_levels)]


def test_one_workspace_for_all_levels():
    """beside the operators, the assembly of all levels keeps its lists (32 bytes
    per tetrahedron, 4 per vertex) and the top level's workspace (64 bytes per
    tetrahedron); a workspace of its own on every level would add a seventh of
    that (48 MB here, the allocations' granularity is below 24 MB)"""
    (rows, sizes), (elements, _) = (_memory_of_operators(r) for r in (2, 0))
    lists = sum(32 * ne + 4 * nv for nv, ne in sizes)
    assert rows - elements <= lists + 64 * sizes[-1][1] + 24 * MB


@pytest.mark.parametrize("warm", [False, True])
def test_elements_where_there_is_no_memory(warm):
    """the allocations fail before the first assembly, or after some: the same
    operator and right-hand side as element by element; with memory again, the
    rows' own"""
    import ugcore_gb300 as ug
    ctx, hier, disc = _disc(ug, 2)
    A, b = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, hier.num_vertices())

    def assembled():
        disc.assemble_linear(A, b)
        return A.export_csr()[2], b.numpy()

    ctx.set_tuning(row_assembly=0)
    elements = assembled()
    ctx.set_tuning(row_assembly=2)
    if warm:
        rows = assembled()
    ctx.set_tuning(scratch_test=1)
    for _ in range(2):
        got = assembled()
        assert np.array_equal(got[0], elements[0]) and np.array_equal(got[1], elements[1])
    ctx.set_tuning(scratch_test=0)
    again = assembled()
    if warm:
        assert np.array_equal(again[0], rows[0]) and np.array_equal(again[1], rows[1])
    assert np.abs(again[0] - elements[0]).max() <= 1e-12 * np.abs(elements[0]).max()
