"""Multi-vector products with rows of many pieces (512 entries each): around the piece count from which the whole CTA
sums a row, around whole tiles of its ring (64 or 32 pieces of 32 columns), and many more long rows than CTAs.

Tolerance: a column's sum of L products, with values and vectors that are exact in the arithmetic's type, is within
(L + 8) * u * sum|products|, u the unit roundoff of the sums (2^-24 or 2^-53)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,vec,u", [("f64", "f64", 2.0 ** -53), ("f32", "f32", 2.0 ** -24)])
@pytest.mark.parametrize("k", [32, 64, 128])
@pytest.mark.parametrize("pieces", [[63, 64, 65, 66, 127, 128, 129, 1, 0], [200, 2, 321, 0, 96, 97],
                                    [2] * 2500 + [70, 3]])
def test_long_rows(storage, vec, u, k, pieces):
    import frovedis_gb300 as fv
    from scipy.sparse import csr_matrix
    rng = np.random.default_rng(len(pieces) + k)
    lens = [max(0, p * 512 - int(rng.integers(0, 2)) * 511) for p in pieces]
    m, n = len(lens), 4096
    off = np.zeros(m + 1, dtype=np.int32)
    off[1:] = np.cumsum(lens)
    idx = rng.integers(0, n, off[-1]).astype(np.int32)
    val = rng.standard_normal(off[-1]).astype(np.float32).astype(np.float64)
    X = rng.standard_normal((n, k)).astype(np.float32)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, idx, val)
        Y = A.spmm(X, storage=storage, vec=vec)
        A.close()
    ref = csr_matrix((val, idx, off), (m, n)) @ X.astype(np.float64)
    mag = csr_matrix((np.abs(val), idx, off), (m, n)) @ np.abs(X.astype(np.float64))
    bound = (np.array(lens)[:, None] + 8) * u * mag + (2.0 ** -24 * np.abs(ref) if vec == "f32" else 0)
    assert np.all(np.abs(Y - ref) <= bound + 1e-300)


@pytest.mark.parametrize("storage,u", [("f64", 2.0 ** -53), ("f32", 2.0 ** -24), ("bf16", 2.0 ** -24)])
@pytest.mark.parametrize("k", [8, 32, 40, 64, 128])
@pytest.mark.parametrize("empty_runs", [False, True])
def test_chunk_edges(storage, u, k, empty_runs):
    """Rows around the 32 entries of a chunk; runs of empty rows that fill whole work items, so that the entries fetched
    ahead belong to a row several items later."""
    import frovedis_gb300 as fv
    from scipy.sparse import csr_matrix
    vec = "f64" if storage == "f64" else "f32"
    rng = np.random.default_rng(k)
    lens = rng.choice([0, 1, 2, 7, 8, 9, 31, 32, 33, 40, 63, 64, 65, 511, 512, 513], 6000)
    if empty_runs:
        lens[rng.random(6000) < 0.5] = 0
        for s in range(0, 6000, 400):
            lens[s:s + 300] = 0
    m, n = len(lens), 3000
    off = np.zeros(m + 1, dtype=np.int32)
    off[1:] = np.cumsum(lens)
    idx = rng.integers(0, n, off[-1]).astype(np.int32)
    val = (rng.integers(-128, 129, off[-1]) / 64.0)  # exact in every storage type
    X = rng.standard_normal((n, k)).astype(np.float32)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, idx, val)
        Y = A.spmm(X, storage=storage, vec=vec)
        A.close()
    ref = csr_matrix((val, idx, off), (m, n)) @ X.astype(np.float64)
    mag = csr_matrix((np.abs(val), idx, off), (m, n)) @ np.abs(X.astype(np.float64))
    bound = (lens[:, None] + 8) * u * mag + (2.0 ** -24 * np.abs(ref) if vec == "f32" else 0)
    assert np.all(np.abs(Y - ref) <= bound + 1e-300)
