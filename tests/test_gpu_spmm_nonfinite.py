"""Multi-vector products with an infinity and a NaN in a row of X that no entry of the matrix reads: rows whose last
chunk of 32 entries is not full must not pick them up from the chunk's padding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("k", [1, 2, 3, 8, 32, 34, 64, 128])
def test_unread_row_of_x(storage, k):
    import frovedis_gb300 as fv
    rng = np.random.default_rng(k)
    m, n = 400, 50
    lens = rng.integers(0, 40, m)
    lens[:34] = np.arange(34)
    off = np.zeros(m + 1, dtype=np.int32)
    off[1:] = np.cumsum(lens)
    idx = np.concatenate([np.sort(rng.choice(np.arange(1, n), c, replace=False)) for c in lens]).astype(np.int32)
    val = rng.integers(1, 9, off[-1]).astype(np.float64)
    X = rng.integers(-8, 9, (n, k)).astype(np.float64)
    X[0] = np.where(np.arange(k) % 2 == 0, np.inf, np.nan)
    dense = np.zeros((m, n))
    for r in range(m):
        dense[r, idx[off[r]:off[r + 1]]] = val[off[r]:off[r + 1]]
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, idx, val)
        Y = A.spmm(X, storage=storage, vec="f64" if storage == "f64" else "f32")
        A.close()
    assert np.array_equal(Y, dense[:, 1:] @ X[1:])  # small whole numbers: exact in every type
