"""The slab-ordered work items of a batched training depend on the training alone, not on the one before: FP64 with 32
models and FP32 with 64 have slabs of the same height, and items of their own."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def test_items_follow_the_storage():
    import frovedis_gb300 as fv
    from frovedis_gb300 import datagen
    off, idx, val, label = datagen.generate(datagen.Spec(m=20_000, n=200, lam=15.0, seed=2))

    def train(A, storage, k):
        n0 = A.ctx.kernel_launches
        fv.logreg_lbfgs_batched(A, label, np.logspace(-4, 0, k), num_iter=2, reg_type="L2", storage=storage)
        return A.ctx.kernel_launches - n0

    with fv.Context(0) as ctx:
        launches = []
        for before in (False, True):
            A = ctx.matrix(20_000, 200, off, idx, val)
            A.prepare("CRS", transpose=True)
            A.add_storage("f32")
            if before:
                train(A, "f64", 32)
            launches.append(train(A, "f32", 64))
            again = train(A, "f32", 64)
            assert again < launches[-1]  # the items are built once
            A.close()
        assert launches[0] == launches[1]
