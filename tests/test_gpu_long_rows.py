"""Row-wise assembly of unstructured simplices (k_fv1_gather.cu) whose blocks of
64 rows hold more values than 48 KB of shared memory: 64 vertices, numbered one
after the other, each the only common corner of as many elements as a row's 256
candidates admit (64 tetrahedra, 193 entries, 99 KB; 85 triangles, 171 entries,
87 KB), against the element kernel.  An entry off the diagonal comes from one
element, a few products of edge vectors: 1e-12 of its row's largest entry; a
diagonal sums up to 85 of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bouquets(elem):
    k, per = (4, 64) if elem == "tet" else (3, 85)
    rng = np.random.default_rng(7)
    hubs, dim = 64, k - 1
    x = [3.0 * np.arange(hubs)[:, None] * np.ones(dim)]
    e, n = [], hubs
    for h in range(hubs):
        for _ in range(per):
            # corners near the coordinate directions of a random frame: no sliver
            q = np.linalg.qr(rng.normal(size=(dim, dim)))[0] + rng.uniform(-0.1, 0.1, (dim, dim))
            x.append(x[0][h] + q)
            e.append([h] + list(range(n, n + dim)))
            n += dim
    return np.vstack(x), np.array(e)


@pytest.mark.parametrize("elem", ["tet", "tri"])
def test_matches_elements(elem):
    import ugcore_gb300 as ug
    x, e = _bouquets(elem)
    one = np.zeros(len(x), np.uint8)
    one[-1] = 1
    got = []
    for rows in (2, 0):
        ctx = ug.Context(0)
        ctx.set_tuning(row_assembly=rows)
        hier = ug.UnstructuredHierarchy.from_arrays(ctx, elem, x, e, dirichlet_vertices=one)
        disc = ug.DomainDiscretization(hier)
        rng = np.random.default_rng(5)
        disc.set_log_diffusion(rng.normal(size=hier.num_elements()))
        disc.set_source(rng.uniform(-1, 1, len(x)))
        A, b = ug.GPUSparseMatrix(ctx), ug.GPUVector(ctx, len(x))
        disc.assemble_linear(A, b)
        stationary = A.export_csr() + (b.numpy(),)
        td = ug.ThetaTimeStep(disc, 0.5)
        td.prepare_step(ug.GPUVector(ctx, len(x)).copy_from(rng.uniform(-1, 1, len(x))), 0.0, 0.05)
        td.assemble_linear(A, b)
        got.append(stationary + (A.export_csr()[2], b.numpy()))
    (rp, ci, va, b0, vt, b1), want = got
    assert rp[64] * 8 > 48 * 1024
    assert np.array_equal(rp, want[0]) and np.array_equal(ci, want[1])
    for v, w in ((va, want[2]), (vt, want[4])):
        row_max = np.maximum.reduceat(np.abs(w), rp[:-1])
        assert np.all(np.abs(v - w) <= 1e-12 * np.repeat(row_max, np.diff(rp)))
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    scale = np.bincount(rows, np.abs(want[2])).max() + np.abs(want[3]).max()
    assert np.abs(b0 - want[3]).max() <= 1e-13 * np.abs(want[3]).max()
    assert np.abs(b1 - want[5]).max() <= 1e-12 * (scale + np.abs(want[5]).max())
