"""The streamed layout of the row panels and the forward head where its shape changes: segments that end on, before and
after a chunk of 4 entries and the 64-entry limit, slices of fewer than 32 segments, empty rows, long rows, and a vector
entry that only the padding could touch.

Tolerances: FP32 sums are 4 chains of at most 16 adds, joined by at most 32 more roundings over the segments, panels and
the product itself (48 * 2^-24 of the sum of magnitudes); a split value is within 2^-33 of its FP64 value and the df64
arithmetic below 2^-40 (2^-32 together)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 1024  # per panel
LENS = [1, 2, 3, 4, 5, 8, 31, 32, 33, 60, 61, 63, 64, 65, 67, 68, 127, 128, 129, 192, 193, 500, 1000]


def _columns(rng, m, copies):
    """Columns with LENS entries in every panel (row 0 stays unused), in CSC form: (row, column) pairs."""
    rows, cols = [], []
    n = 0
    for _ in range(copies):
        for k in LENS:
            for p0 in range(0, m, ROWS):
                hi = min(m, p0 + ROWS)
                k2 = min(k, hi - max(p0, 1))
                r = np.sort(rng.choice(np.arange(max(p0, 1), hi), k2, replace=False))
                rows.append(r)
                cols.append(np.full(k2, n))
            n += 1
    return np.concatenate(rows), np.concatenate(cols), n


def _crs(rows, cols, m, n, rng):
    o = np.lexsort((cols, rows))
    rows, cols = rows[o], cols[o]
    off = np.zeros(m + 1, dtype=np.int32)
    off[1:] = np.cumsum(np.bincount(rows, minlength=m))
    return off, cols.astype(np.int32), rng.standard_normal(len(cols))


@pytest.mark.parametrize("storage", ["f32", "bf16", "split"])
@pytest.mark.parametrize("m,copies", [(2 * ROWS, 1), (3 * ROWS + 7, 3)])
def test_panels(storage, m, copies):
    import frovedis_gb300 as fv
    import oracle
    rng = np.random.default_rng(copies)
    rows, cols, n = _columns(rng, m, copies)
    off, idx, val = _crs(rows, cols, m, n, rng)
    if storage != "split":
        val = val.astype(np.float32).astype(np.float64)
    if storage == "bf16":
        val = ((val.astype(np.float32).view(np.uint32) & 0xFFFF0000).view(np.float32)).astype(np.float64)
    x = rng.standard_normal(m)
    if storage != "split":
        x = x.astype(np.float32).astype(np.float64)
    t = oracle.transpose(oracle.CRS(m, n, off, idx, val))
    ta = oracle.transpose(oracle.CRS(m, n, off, idx, np.abs(val)))
    want, mag = oracle.spmv(t, x), oracle.spmv(ta, np.abs(x))
    x[0] = np.inf  # no entry of the matrix reads it
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, idx, val)
        A.set_panels(ROWS, 1.0)
        y = A.trans_mv(x, storage=storage, vec="f64" if storage == "split" else "f32")
        assert A.panel_info()[2] == n
        A.close()
    bar = 2.0 ** -32 if storage == "split" else 48 * 2.0 ** -24
    assert np.all(np.abs(y - want) <= bar * mag)


@pytest.mark.parametrize("storage", ["f32", "split"])
@pytest.mark.parametrize("m", [5, 700])
def test_head(storage, m):
    """Rows of every length in the head (at most 3,000 columns wide), empty rows among them."""
    import frovedis_gb300 as fv
    import oracle
    rng = np.random.default_rng(m)
    n = 3000
    lens = rng.choice([0] + LENS + [2900], m)
    off = np.zeros(m + 1, dtype=np.int32)
    off[1:] = np.cumsum(lens)
    idx = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens]).astype(np.int32)
    val = rng.standard_normal(len(idx)).astype(np.float32).astype(np.float64)
    w = rng.standard_normal(n).astype(np.float32).astype(np.float64)
    label = rng.standard_normal(m).astype(np.float32).astype(np.float64)
    a = oracle.CRS(m, n, off, idx, val)
    go, lo = oracle.logreg_eval(a, label, w, loss="linear")
    mag = oracle.spmv(oracle.CRS(m, n, off, idx, np.abs(val)), np.abs(w)) + np.abs(label)
    gm = oracle.spmv(oracle.transpose(oracle.CRS(m, n, off, idx, np.abs(val))), mag)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, idx, val)
        A.set_head(2500)
        A.set_panels(0)
        g, loss = fv.glm_eval(A, label, w, storage=storage, loss="linear")
        assert A.head_info()[0] == 2500
        A.close()
    # a residual's error (first bound of the module) enters the gradient once more, with the same kind of sum on top
    bar = (2.0 ** -32 if storage == "split" else 48 * 2.0 ** -24) * 3
    assert np.all(np.abs(g[:-1] - go[:-1]) <= bar * gm)
    assert abs(loss - lo) <= bar * (mag ** 2).sum()
