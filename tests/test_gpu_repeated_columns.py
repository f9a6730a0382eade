"""CRS -> diagonals (k_dia_fill) of rows that name a column twice: the last value
of the row stays, whichever of the threads of a row it falls to (rows of 3 to 27
entries, the repetition next to the first one, in the middle or at the end).
Whole numbers, so that the products are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", [1, 2, -1])
@pytest.mark.parametrize("width,n", [(1, 64), (3, 200), (13, 500)])
def test_last_value_stays(width, n, where):
    import ugcore_gb300 as ug
    ctx = ug.Context(0)
    rng = np.random.default_rng(width)
    rp, ci, want = [0], [], np.zeros((n, n))
    va = []
    for r in range(n):
        c = [r + o for o in range(-width, width + 1) if 0 <= r + o < n]
        v = list(rng.integers(1, 100, len(c) + 1).astype(float))
        at = len(c) if where < 0 else where
        c.insert(at, c[0])
        for cc, vv in zip(c, v):
            want[r, cc] = vv
        ci += c
        va += v
        rp.append(len(ci))
    A = ug.GPUSparseMatrix(ctx).set_csr(rp, ci, va)
    x = rng.integers(-50, 50, n).astype(float)
    xv, yv = ug.GPUVector(ctx, n).copy_from(x), ug.GPUVector(ctx, n)
    A.apply(yv, xv)
    assert np.array_equal(yv.numpy(), want @ x)
