"""Kernels chosen by size, on both sides of each line: long rows one or four to a warp (4,864 on 152 SMs), the L-BFGS
direction on few or many CTAs (32,768 model elements), the trial loop of the batched trainer, and the column sums of
one group of CTAs or several.

Tolerances.  Products: (L + 8) * 2^-53 * sum|products| for a row of L products.  Trainings: the parity bar of the
trainers, loss 1e-6 and weights 1e-5 relative, with the same iteration count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlong", [1, 4863, 4864, 4865, 6000])
def test_long_row_sums(nlong):
    import frovedis_gb300 as fv
    from scipy.sparse import csr_matrix
    rng = np.random.default_rng(nlong)
    lens = rng.integers(513, 700, nlong)
    lens[:: max(nlong // 3, 1)] = 512 * 33 + 5  # more pieces than the lanes of a quarter warp take at once
    lens = np.insert(lens, rng.integers(0, nlong + 1, 200), rng.integers(0, 40, 200))
    m, n = len(lens), 3000
    off = np.zeros(m + 1, np.int32)
    off[1:] = np.cumsum(lens)
    idx = rng.integers(0, n, off[-1]).astype(np.int32)
    val, x = rng.standard_normal(off[-1]), rng.standard_normal(n)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, idx, val)
        y = A.spmv(x)
        A.close()
    mag = csr_matrix((np.abs(val), idx, off), (m, n)) @ np.abs(x)
    assert np.all(np.abs(y - csr_matrix((val, idx, off), (m, n)) @ x) <= 2 * (lens + 8) * 2.0 ** -53 * mag)


def _problem(m, n, seed):
    rng = np.random.default_rng(seed)
    lens = rng.integers(5, 40, m)
    off = np.zeros(m + 1, np.int32)
    off[1:] = np.cumsum(lens)
    idx = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens]).astype(np.int32)
    val = rng.standard_normal(off[-1])
    return off, idx, val, np.where(rng.random(m) < 0.5, 1.0, -1.0)


@pytest.mark.parametrize("n", [50, 4095, 32766, 32767, 32768, 70000])
@pytest.mark.parametrize("intercept", [False, True])
def test_direction_sizes(n, intercept):
    import frovedis_gb300 as fv
    import oracle
    m = 1500
    off, idx, val, lab = _problem(m, n, n)
    kw = dict(num_iter=12, hist_size=5, reg_type="L2", reg_param=1e-2, intercept=intercept)
    ref = oracle.logreg_lbfgs(oracle.CRS(m, n, off, idx, val), lab, w0=np.zeros(n), b0=0.0, tol=1e-9, **kw)
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, idx, val)
        r = fv.logreg_lbfgs(A, lab, w0=np.zeros(n), b0=0.0, convergence_tol=1e-9, **kw)
        A.close()
    assert r["n_iter"] == ref["n_iter"]
    assert abs(r["loss"] - ref["loss"]) <= 1e-6 * abs(ref["loss"])
    assert np.linalg.norm(r["w"] - ref["w"]) <= 1e-5 * np.linalg.norm(ref["w"])


@pytest.mark.parametrize("n,k", [(50, 1), (50, 5), (7000, 3), (9000, 64), (300, 100), (5000, 256)])
def test_batched_sizes(n, k):
    """From one CTA of column sums to several groups of 32, one to 256 models; the regularisation values make the
    models take different numbers of trials and stop at different iterations."""
    import frovedis_gb300 as fv
    import oracle
    m = 700
    off, idx, val, lab = _problem(m, n, n + k)
    val *= 3.0
    lam = np.geomspace(1e-4, 0.3, k)
    kw = dict(num_iter=9, hist_size=3, reg_type="L2")
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, n, off, idx, val)
        r = fv.logreg_lbfgs_batched(A, lab, lam, w0=np.zeros((k, n)), convergence_tol=1e-3, **kw)
        A.close()
    a = oracle.CRS(m, n, off, idx, val)
    for j in sorted({0, k // 2, k - 1}):
        ref = oracle.logreg_lbfgs(a, lab, w0=np.zeros(n), reg_param=float(lam[j]), tol=1e-3, **kw)
        assert r["n_iter"][j] == ref["n_iter"]
        assert abs(r["loss"][j] - ref["loss"]) <= 1e-6 * abs(ref["loss"])
        assert np.linalg.norm(r["w"][j] - ref["w"]) <= 1e-5 * max(np.linalg.norm(ref["w"]), 1e-30)
