"""A warp reads several consecutive columns (or smoothing rows) as one stretch of
entries.  Products with A and its transpose against a dense product: columns
with no entry, one, a batch's ends (255 to 257), more than a batch, all rows;
fewer columns than warps and many more."""
import numpy as np
import pytest

from fmt2d_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol,nrow", [(1, 5), (31, 300), (4737, 300), (60001, 777)])
def test_products_of_any_column_length(ncol, nrow):
    from fmt2d_b200.api import Fmt2d
    rng = np.random.default_rng(ncol)
    few = rng.integers(0, 4, ncol)
    for j, n in enumerate((255, 256, 257, 0, 300, 0, 0, 1, 64, 33)):
        if 3 * j < ncol:
            few[3 * j] = n
    few = np.minimum(few, nrow)
    few[-1] = nrow
    col = np.repeat(np.arange(ncol), few)
    row = np.concatenate([rng.permutation(nrow)[:n] for n in few])
    order = np.lexsort((col, row))
    row, col = row[order], col[order]
    val = rng.normal(size=col.size)
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=nrow))]) + 1
    g = Fmt2d(0).upload(synth.small_model())
    g.set_frechet(nrow, ncol, rp.astype(np.int32), (col + 1).astype(np.int32), val)
    x, y = rng.normal(size=ncol), rng.normal(size=nrow)
    ax, aty = g.spmv(x, transpose=False), g.spmv(y, transpose=True)
    # each sum of n products is within n rounding errors of the sum of their sizes
    eps = 2.0 ** -52
    for got, idx, terms, n in ((ax, row, val * x[col], nrow), (aty, col, val * y[row], ncol)):
        want = np.bincount(idx, weights=terms, minlength=n)
        size = np.bincount(idx, weights=np.abs(terms), minlength=n)
        cnt = np.bincount(idx, minlength=n)
        assert np.all(np.abs(got - want) <= 2.0 * eps * cnt * size)
    g.close()
