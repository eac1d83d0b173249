"""Which matrices get row panels by themselves: from 90,112 rows on (22 panels of 4,096), where below the plain product
takes half the time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,panels", [(78_000, 0), (90_111, 0), (90_112, 22), (100_000, 25)])
def test_shortest_matrix(m, panels):
    import frovedis_gb300 as fv
    n, k = 40, 4
    off = np.arange(m + 1, dtype=np.int32) * k
    idx = ((np.arange(m)[:, None] + np.arange(k) * 10) % n).astype(np.int32)
    idx.sort(axis=1)
    val = np.ones((m, k), dtype=np.float32)
    x = (np.arange(m) % 7 - 3).astype(np.float32)
    want = np.bincount(idx.ravel(), weights=np.repeat(x, k).astype(np.float64), minlength=n)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, idx.ravel(), val.ravel())
        y = A.trans_mv(x, storage="f32", vec="f32")
        info = A.panel_info()
        A.close()
    assert info[1] == panels and (info[0] == 4096 if panels else info[0] == 0)
    assert np.array_equal(y, want)  # small whole numbers
