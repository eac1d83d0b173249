"""The FP64 logistic row over its ranges: margins around 0, at every interval of the exponential's and the logarithm's
tables, around the thresholds at 18 and where the exponential leaves the tables (700) and FP64 (745).

Tolerance: exp and log are within 0.52 and the quotient within 0.5 of a unit in the last place (measured against
extended precision); 1 + e rounds once.  d: exp (0.52), 1 + e (0.5), the quotient (0.5), the product with the entry
(0.5), and dividing it out again (0.5): under 3 units.  The loss of a row: exp's error times e, the rounding of 1 + e
and the logarithm's, 2 units of max(loss, 2^-53) at most, plus the compensated sum's last rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _margins(kind, rng):
    if kind == "tables":  # around every multiple of ln 2 / 256 up to 18, and random ones between
        k = np.arange(1, 6600) * (np.log(2.0) / 256)
        return np.concatenate([k, k * (1 + 1e-15), k * (1 - 1e-15), rng.uniform(0, 18, 4000)])
    if kind == "tiny":
        return np.concatenate([2.0 ** -np.arange(1.0, 1000.0, 7.0), [5e-324, 2.2e-308]])
    if kind == "threshold":
        return np.concatenate([18 + np.arange(-40, 41) * 2.0 ** -48, rng.uniform(17, 19, 200)])
    return np.concatenate([rng.uniform(19, 690, 500), 700 + np.arange(-40, 41) * 2.0 ** -43, [708.0, 720.0, 744.0]])


@pytest.mark.parametrize("kind", ["tables", "tiny", "threshold", "far"])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_row(kind, sign):
    import frovedis_gb300 as fv
    z = sign * _margins(kind, np.random.default_rng(5))
    z = z[z != 0]
    m = len(z)
    off, idx = np.arange(m + 1, dtype=np.int32), np.arange(m, dtype=np.int32)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, m, off, idx, z)
        g, loss = fv.logreg_eval(A, np.ones(m), np.ones(m))
        A.close()
    t = np.asarray(z, np.longdouble)
    e = np.exp(-np.abs(t))
    losses = np.where(t > 18, e, np.where(t < -18, -t, np.maximum(-t, 0) + np.log1p(e)))
    d = -np.where(t > 18, e, np.where(t < -18, 1, np.where(t > 0, e, 1) / (1 + e)))
    prod = t * d
    ok = np.abs(prod) > 1e-290  # results that are not subnormal
    assert np.all(np.abs(g[:m] - prod)[ok] <= 4 * 2.0 ** -52 * np.abs(prod)[ok])
    assert abs(loss - losses.sum()) <= 2 * 2.0 ** -52 * (np.maximum(losses, 2.0 ** -53).sum()) + m * 2.0 ** -53


def test_no_number():
    import frovedis_gb300 as fv
    for v in (np.nan, np.inf, -np.inf):
        with fv.Context(0) as ctx:
            A = ctx.matrix(1, 1, np.array([0, 1], np.int32), np.zeros(1, np.int32), np.array([v]))
            g, loss = fv.logreg_eval(A, np.ones(1), np.ones(1))
            A.close()
        if np.isnan(v):
            assert np.isnan(loss) and np.isnan(g[0])
        elif v > 0:
            assert loss == 0.0
        else:
            assert np.isnan(loss)  # an infinite loss: the compensated sum's correction is infinity minus infinity
