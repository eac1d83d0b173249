"""The batched trainer at the library's default number of iterations: one graph with a trial loop for each of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iters", [1, 1000])
def test_default_iterations(iters):
    import frovedis_gb300 as fv
    from frovedis_gb300 import datagen
    assert fv.glm_params().num_iteration == 1000
    off, idx, val, label = datagen.generate(datagen.Spec(m=3000, n=200, lam=15.0, seed=1))
    lam = [1e-3, 1e-1]
    kw = dict(num_iter=iters, reg_type="L2", convergence_tol=0.0)
    with fv.Context(0) as ctx:
        A = ctx.matrix(3000, 200, off, idx, val)
        r = fv.logreg_lbfgs_batched(A, label, lam, **kw)
        one = [fv.logreg_lbfgs(A, label, reg_param=x, **kw) for x in lam]
        A.close()
    assert list(r["n_iter"]) == [iters] * 2
    for loss, s in zip(r["loss"], one):
        # near the minimum the losses of two summation orders wander within the line search's tolerance of 1e-4
        assert abs(loss - s["loss"]) <= 1e-4 * abs(s["loss"])
