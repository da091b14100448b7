"""A matrix that did not fit leaves no matrix behind: products and solves say so,
instead of running on half of it or on the column runs of the one before; the
next matrix that fits is as good as ever."""
import numpy as np
import pytest

from fmt2d_b200 import synth

pytestmark = pytest.mark.gpu


def test_no_matrix_after_a_failed_set():
    import torch
    from fmt2d_b200._native import Fmt2dError
    from fmt2d_b200.api import Fmt2d
    rng = np.random.default_rng(1)

    def rows(nrow, ncol, per):
        rp = (1 + per * np.arange(nrow + 1)).astype(np.int32)
        col = (1 + rng.integers(0, ncol, nrow * per)).astype(np.int32)
        return nrow, ncol, rp, col, rng.normal(size=nrow * per)

    g = Fmt2d(0).upload(synth.small_model())
    small = rows(300, 60000, 64)
    g.set_frechet(*small)
    y = rng.normal(size=300)
    want = g.spmv(y, transpose=True)
    big = rows(40000, 5000, 200)          # 96 MB as rows, as much again as columns
    free, _ = torch.cuda.mem_get_info()
    fill = torch.empty(free - (140 << 20), dtype=torch.uint8, device="cuda")
    with pytest.raises(Fmt2dError, match="allocation"):
        g.set_frechet(*big)
    with pytest.raises(Fmt2dError, match="no matrix"):
        g.spmv(y, transpose=True)
    with pytest.raises(Fmt2dError, match="no matrix"):
        g.gtg_diag()
    del fill
    torch.cuda.empty_cache()
    g.set_frechet(*small)
    assert g.spmv(y, transpose=True).tobytes() == want.tobytes()
    g.close()
