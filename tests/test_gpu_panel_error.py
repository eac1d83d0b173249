"""How far the FP32 sums of the row panels are from the FP64 product, on columns with thousands of entries a panel.

A rounding of a number spread over a binade is 0.408 * 2^-24 of it (root mean square), and a chain of L adds of random
signs makes L / 2 of them in the sum's own size (as variances).  An entry's product makes 1, its chain of 8 adds 4, the
join of a segment's 8 chains 3, the rounding of a panel's sum 1 and that of the result 1: 10 in all, 3.2 roundings.
Chains of 16 adds and plain sums over the segments would make 8 + 2 + 2.8 + 5 and the same 2: 20, 4.5 roundings.  The
bar lies between, at 3.8; 200 columns put the measured value within a few percent of its expectation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_error_of_long_columns(storage):
    import frovedis_gb300 as fv
    rng = np.random.default_rng(7)
    m, n = 32_000, 200
    mask = rng.random((m, n)) < 0.9
    off = np.zeros(m + 1, dtype=np.int32)
    off[1:] = np.cumsum(mask.sum(1))
    rows, cols = np.nonzero(mask)
    val = rng.standard_normal(len(cols)).astype(np.float32)
    if storage == "bf16":
        val = (val.view(np.uint32) & 0xFFFF0000).view(np.float32)
    x = rng.standard_normal(m).astype(np.float32)
    want = np.bincount(cols, weights=val.astype(np.float64) * x[rows].astype(np.float64), minlength=n)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, cols.astype(np.int32), val.astype(np.float64))
        A.set_panels(12_800, 1.0)
        y = A.trans_mv(x, storage=storage, vec="f32").astype(np.float64)
        assert A.panel_info()[2] == n
        A.close()
    err = np.linalg.norm(y - want) / np.linalg.norm(want)
    assert err <= 3.8 * 0.408 * 2.0 ** -24, err
