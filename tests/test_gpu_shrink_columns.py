"""Shrink SGD with any number of columns: rank 0's column count is kept beside the column marks, and odd numbers of them
leave it no 8-byte place at their end."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 300, 301])
def test_number_of_columns(n):
    import frovedis_gb300 as fv
    rng = np.random.default_rng(n)
    m = 1500
    lens = rng.integers(0, min(n, 12) + 1, m)
    off = np.zeros(m + 1, dtype=np.int32)
    off[1:] = np.cumsum(lens)
    idx = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens]).astype(np.int32)
    a = oracle.CRS(m, n, off, idx, rng.standard_normal(off[-1]))
    label = np.where(rng.random(m) < 0.5, 1.0, -1.0)
    splits = [0, 700, m]
    kw = dict(num_iter=5, alpha=0.01, mini_batch_fraction=0.5, reg_type="L2", reg_param=1e-2, intercept=True)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, a.off, a.idx, a.val)
        r = fv.logreg_shrink_sgd(A, label, row_splits=splits, **kw)
        A.close()
    ro = oracle.logreg_sgd(a, label, shrink=True, splits=splits, **kw)
    assert r["n_iter"] == ro["n_iter"]
    assert abs(r["loss"] - ro["loss"]) <= 1e-6 * abs(ro["loss"])
    assert np.max(np.abs(r["w"] - ro["w"])) <= 1e-5 * max(1.0, np.max(np.abs(ro["w"])))
