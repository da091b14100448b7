"""A^T y with so many columns that a lane adds up a whole column, in trees of eight
whose sums' additions carry their roundings along.  Columns of 60 positive
products: the products and the trees round parts of the sum that are small beside
it, the sum itself is rounded once: in the root mean square less than one rounding
unit (one product after the other, 60 partial sums are rounded: about two)."""
import numpy as np
import pytest

from fmt2d_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol,per", [(320000, 60), (40000, 61)])
def test_transposed_product_error(ncol, per):
    from fmt2d_b200.api import Fmt2d
    rng = np.random.default_rng(ncol)
    nrow = per * 4
    # column j holds rows (j + 4 i) mod nrow; as rows: ascending columns
    col = np.repeat(np.arange(ncol), per)
    row = (col + 4 * np.tile(np.arange(per), ncol)) % nrow
    order = np.argsort(row, kind="stable")
    val = rng.uniform(0.5, 1.5, ncol * per)
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=nrow))])
    g = Fmt2d(0).upload(synth.small_model())
    g.set_frechet(nrow, ncol, rp.astype(np.int32), col[order].astype(np.int32), val[order],
                  index_base=0)
    y = rng.uniform(0.5, 1.5, nrow)
    got = g.spmv(y, transpose=True)
    terms = val.astype(np.longdouble) * y[row]
    want = np.add.reduceat(terms, np.arange(0, ncol * per, per))
    err = ((got - want) / want).astype(np.float64)
    assert np.sqrt(np.mean(err ** 2)) <= 2.0 ** -53
    # a sum that is not finite stays what plain additions give
    y[1] = np.inf
    hit = np.bincount(col, weights=(row == 1), minlength=ncol) > 0
    got = g.spmv(y, transpose=True)
    assert np.all(np.isposinf(got[hit])) and np.all(np.isfinite(got[~hit]))
    g.close()
