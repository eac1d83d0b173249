"""Multi-vector products on both sides of the rules that choose how their gathers are issued: rows of fewer than 7 (or
15) entries on average, and columns scattered over more than 64 MB of X.  Whole numbers, so every order of the sums
gives the same result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("k", [8, 32, 40, 64])
@pytest.mark.parametrize("n,avg,scattered", [(3000, 5, True), (3000, 9, False), (3000, 20, False), (300_000, 5, True),
                                             (300_000, 20, True), (300_000, 20, False)])
def test_both_sides(storage, k, n, avg, scattered):
    import frovedis_gb300 as fv
    from scipy.sparse import csr_matrix
    rng = np.random.default_rng(n + avg + k)
    m = 4000
    lens = rng.integers(0, 2 * avg + 1, m)
    lens[:5] = [0, 1, 600, 33, 0]
    off = np.zeros(m + 1, dtype=np.int32)
    off[1:] = np.cumsum(lens)
    if scattered:
        idx = rng.integers(0, n, off[-1])
    else:  # a few columns hold most entries
        idx = np.minimum((n * rng.random(off[-1]) ** 40).astype(np.int64), n - 1)
    idx = idx.astype(np.int32)
    val = rng.integers(1, 5, off[-1]).astype(np.float64)
    X = rng.integers(-4, 5, (n, k)).astype(np.float32)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, idx, val)
        Y = A.spmm(X, storage=storage, vec="f64" if storage == "f64" else "f32")
        A.close()
    assert np.array_equal(Y, csr_matrix((val, idx, off), (m, n)) @ X.astype(np.float64))
