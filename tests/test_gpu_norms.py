"""Gradient norms of the L-BFGS trainers beyond the ordinary range: sizes whose squares leave FP64, NaN and zeros.  The
norm scales by the largest magnitude that is a number, so a gradient of NaN and zeros has norm 0 and ends the training.

The sizes: three rows of one feature v with labels 1, 1, -1 and zero initial weight.  A tiny v leaves the margins at 0
and the gradient at -v/2; a huge one turns every margin's exponential to 0 or infinity and the gradient to +v.  The rms
over the feature and the (empty) intercept is that over sqrt(2): 0.3536 v and 0.7071 v; a tolerance 1% below or above
decides whether the training stops after its first iteration."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _iterations(batched, vals, lab, tol):
    import frovedis_gb300 as fv
    m = len(vals)
    off, idx = np.arange(m + 1, dtype=np.int32), np.zeros(m, np.int32)
    kw = dict(num_iter=2, convergence_tol=tol, storage="f64")
    with fv.Context(0) as ctx:
        A = ctx.matrix(m, 1, off, idx, np.array(vals))
        if batched:
            r = fv.logreg_lbfgs_batched(A, lab, [0.0, 0.0], w0=np.zeros((2, 1)), **kw)
            it = {int(x) for x in r["n_iter"]}
        else:
            it = {int(fv.logreg_lbfgs(A, lab, w0=np.zeros(1), **kw)["n_iter"])}
        A.close()
    assert len(it) == 1
    return it.pop()


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("v,rms", [(1e-300, 0.35355339), (1e-160, 0.35355339), (1e160, 0.70710678), (1e300, 0.70710678)])
def test_tiny_and_huge_gradients(batched, v, rms):
    lab = np.array([1.0, 1.0, -1.0])
    assert _iterations(batched, [v] * 3, lab, 0.99 * rms * v) == 2
    assert _iterations(batched, [v] * 3, lab, 1.01 * rms * v) == 1


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("vals", [[np.nan], [np.nan, 1.0], [0.0], [np.inf]])
def test_gradients_without_a_number(batched, vals):
    assert _iterations(batched, vals, np.ones(len(vals)), 1e-300) == 1
