"""The FP64 CRS kernel at the sizes where its item layout changes: rows that end on, before and after a lane's chunk,
empty rows, items of every chunk length, items full of short rows, pieces of long rows.

Tolerance: a row's sum of L products in any order differs from the oracle's by at most (L + 8) * 2^-53 times the sum of
the products' magnitudes (one rounding per multiply-add and at most 8 joins)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(kind, rng):
    if kind == "every span":  # one item of each number of entries (a tile-long row closes the item before it)
        out = []
        for span in range(1, 512, 7):
            left = span
            while left:
                n = int(rng.integers(0, min(left, 60) + 1))
                out.append(n)
                left -= n
            out.append(512)
        return out
    if kind == "chunk edges":  # row ends around multiples of the 16 entries of a lane
        return [int(n) for n in rng.choice([1, 15, 16, 17, 31, 32, 33, 48], 700)]
    if kind == "short and empty":  # the row limit of an item before its entry limit
        return [int(n) for n in rng.choice([0, 0, 1, 2], 3000)]
    if kind == "long":  # pieces, and neighbours of pieces
        return [513, 1, 0, 512, 511, 1024, 2, 5000, 0, 40000, 3]
    return [0] * 300  # nothing stored


@pytest.mark.parametrize("kind", ["every span", "chunk edges", "short and empty", "long", "empty"])
@pytest.mark.parametrize("trans", [False, True])
def test_fp64_products(kind, trans):
    import frovedis_gb300 as fv
    import oracle
    rng = np.random.default_rng(7)
    lens = np.array(_rows(kind, rng))
    m, n = len(lens), 40000
    off = np.zeros(m + 1, dtype=np.int32)
    off[1:] = np.cumsum(lens)
    idx = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens] + [np.zeros(0, int)]).astype(np.int32)
    val = rng.standard_normal(len(idx))
    ref, mag = oracle.CRS(m, n, off, idx, val), oracle.CRS(m, n, off, idx, np.abs(val))
    if trans:
        ref, mag = oracle.transpose(ref), oracle.transpose(mag)
    x = rng.standard_normal(m if trans else n)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, idx, val)
        y = A.trans_mv(x) if trans else A.spmv(x)
        A.close()
    longest = max(int(lens.max()), m if trans else 0)
    bound = (longest + 8) * 2.0 ** -53 * oracle.spmv(mag, np.abs(x))
    assert np.all(np.abs(y - oracle.spmv(ref, x)) <= bound)


def _logistic(z, y):
    """Loss and derivative of gradient.hpp:24-50 per row, in extended precision."""
    t = np.asarray(y, np.longdouble) * z
    e = np.exp(-np.abs(t))
    loss = np.where(t > 18, e, np.where(t < -18, -t, np.maximum(-t, 0) + np.log1p(e)))
    d = np.where(t > 18, e, np.where(t < -18, 1, np.where(t > 0, e, 1) / (1 + e)))
    return loss, -y * d


@pytest.mark.parametrize("m", [1, 31, 257, 5000])
def test_fp64_logistic_rows(m):
    """The loss rows after the product: margins in every branch, with and without intercept and weights."""
    import frovedis_gb300 as fv
    rng = np.random.default_rng(m)
    off = np.arange(m + 1, dtype=np.int32)
    idx = np.zeros(m, dtype=np.int32)
    val = rng.choice([-800.0, -40.0, -18.0, -1.0, -1e-9, 0.0, 1e-9, 1.0, 17.9, 18.0, 18.1, 40.0, 800.0], m)
    label = rng.choice([-1.0, 1.0], m)
    sw = rng.uniform(0.5, 2.0, m)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, 1, off, idx, val)
        for kw in ({}, {"b": 0.25, "intercept": True}, {"sample_weight": sw}):
            g, loss = fv.logreg_eval(A, label, np.ones(1), **kw)
            losses, d = _logistic(val + kw.get("b", 0.0), label)
            w = kw.get("sample_weight", np.ones(m))
            lo = losses.sum()
            # a handful of roundings per row: exp, log and the quotient are good to a few 2^-53
            scale = np.abs(val * (sw if "sample_weight" in kw else 1.0)).sum() + m
            assert abs(loss - lo) <= 16 * 2.0 ** -53 * (abs(lo) + m)
            assert abs(g[0] - (val * d * w).sum()) <= 16 * 2.0 ** -53 * scale * 2
            assert abs(g[1] - ((d * w).sum() if "b" in kw else 0.0)) <= 16 * 2.0 ** -53 * scale * 2
        A.close()
