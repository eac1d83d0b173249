"""A call whose device allocations fail, whichever of them fails first: it reports FVG_ERR_OUT_OF_MEMORY and leaves
nothing half made on the matrix, so that the same call made again gives what it gives on a matrix that never failed.
The failures are injected on the host; no kernel runs on a buffer that was not allocated."""
import numpy as np
import pytest

import oracle

fv = pytest.importorskip("frovedis_gb300")

pytestmark = pytest.mark.gpu

FVG_ERR_OUT_OF_MEMORY = 5


def _every_failure(make, call):
    """call(A) on matrices from make(): the n-th allocation fails, for every n until none is left to fail."""
    inject = fv.load().fvg_debug_inject_alloc_failure
    A = make()
    good = call(A)
    A.close()
    n = 0
    while True:
        A = make()
        inject(n)
        try:
            got = call(A)
        except fv.FvgError as e:
            assert e.code == FVG_ERR_OUT_OF_MEMORY, (n, str(e))
            got = None
        finally:
            inject(-1)
        done = got is not None  # the call needs no more than n allocations
        again = call(A)
        for a, b in zip(again, good):
            assert np.array_equal(a, b), n
        A.close()
        if done:
            return n
        n += 1


def _matrix(m=2000, n=300, lam=15.0, seed=4):
    from frovedis_gb300 import datagen
    off, idx, val, label = datagen.generate(datagen.Spec(m=m, n=n, lam=lam, seed=seed))
    return oracle.CRS(m, n, off, idx, val), label


@pytest.mark.parametrize("storage", ["f32", "bf16", "split"])
def test_panel_and_head_layouts(storage):
    a, label = _matrix()
    w = np.random.default_rng(1).standard_normal(a.n) * 0.2
    # the most frequent column has more than 64 entries in a panel of 1000 rows: sums of several segments
    assert np.bincount(a.idx[:a.off[1000]], minlength=a.n).max() > 64

    with fv.Context(0) as ctx:
        def make():
            A = ctx.matrix(a.m, a.n, a.off, a.idx, a.val)
            A.prepare("CRS", transpose=True)
            A.set_panels(1000, 1.0)
            A.set_head(64)
            return A

        def call(A):
            g, loss = fv.logreg_eval(A, label, w, b=0.3, intercept=True, storage=storage)
            assert A.panel_info()[2] > 0 and A.head_info()[0] == 64
            return [g, loss]

        assert _every_failure(make, call) > 30


@pytest.mark.parametrize("fmt", ["CRS", "ELL", "JDS", "HYBRID"])
def test_first_use_of_a_format(fmt):
    """The transposed copy and the format's own layouts, built by the call itself; also the bytes the matrix reports."""
    a, _ = _matrix(m=700, n=90, lam=8.0)
    x = np.random.default_rng(2).standard_normal(a.n)
    r = np.random.default_rng(3).standard_normal(a.m)
    with fv.Context(0) as ctx:
        def call(A):
            y = [A.spmv(x, fmt=fmt), A.trans_mv(r, fmt=fmt)]
            return y + [A.device_bytes]

        assert _every_failure(lambda: ctx.matrix(a.m, a.n, a.off, a.idx, a.val), call) > 10


@pytest.mark.parametrize("what", ["batched", "multinomial", "probability", "sgd"])
def test_first_use_by_a_trainer(what):
    a, label = _matrix(m=600, n=80, lam=8.0)
    kinds = (np.arange(a.m) % 3).astype(np.float64)
    W = np.random.default_rng(5).standard_normal((a.n, 3))

    def call(A):
        if what == "batched":
            r = fv.logreg_lbfgs_batched(A, label, [1e-3, 1e-1], num_iter=3, reg_type="L2")
            return [r["w"], r["loss"]]
        if what == "multinomial":
            r = fv.multinomial_lbfgs(A, kinds, 3, num_iter=2, reg_type="L2", reg_param=1e-3)
            return [r["W"], r["loss"]]
        if what == "probability":
            return [fv.multinomial_probability(A, W, np.zeros(3))]
        r = fv.logreg_sgd(A, label, num_iter=2, alpha=0.01, mini_batch_fraction=0.5)
        return [r["w"], r["loss"]]

    with fv.Context(0) as ctx:
        assert _every_failure(lambda: ctx.matrix(a.m, a.n, a.off, a.idx, a.val), call) > 2


def test_next_call_after_a_real_failure():
    """More memory than any device has: refused by the driver itself, which keeps the error until it is read."""
    a, _ = _matrix(m=50, n=40, lam=5.0)
    x = np.random.default_rng(6).standard_normal(a.n)
    n, k = 2_000_000_000, 128
    with fv.Context(0) as ctx:
        A = ctx.matrix(a.m, a.n, a.off, a.idx, a.val)
        good = A.spmv(x)
        W = ctx.matrix(1, n, np.array([0, 1], dtype=np.int32), np.array([7], dtype=np.int32), np.ones(1))
        for _ in range(2):
            with pytest.raises(fv.FvgError) as e:
                # the FP32 copy of X (1 TB) is allocated before X is looked at; Y is never written
                W.spmm_device(16, k, 16, storage="f32", vec="f64")
            assert e.value.code == FVG_ERR_OUT_OF_MEMORY
            assert np.array_equal(A.spmv(x), good)
        W.close()
        A.close()
