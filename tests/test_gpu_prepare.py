"""What fvg_matrix_prepare leaves for the first call: with the storages added before it, the first evaluation in one of
them allocates nothing more on the matrix."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _matrix(m=3000, n=300):
    from frovedis_gb300 import datagen
    off, idx, val, label = datagen.generate(datagen.Spec(m=m, n=n, lam=15.0, seed=3))
    return oracle.CRS(m, n, off, idx, val), label


@pytest.mark.parametrize("storages", [["f32"], ["bf16"], ["f32", "bf16"], ["split", "f32"], ["f32", "split", "bf16"]])
def test_added_storages_are_ready(storages):
    import frovedis_gb300 as fv
    a, label = _matrix()
    w = np.linspace(-0.5, 0.5, a.n)
    with fv.Context(0) as ctx:
        A = ctx.matrix(a.m, a.n, a.off, a.idx, a.val)
        A.set_panels(1000, 1.0)
        A.set_head(64)
        for s in storages:
            A.add_storage(s)
        A.prepare("CRS", transpose=True)
        used = A.device_bytes
        for s in storages:
            if s != "split":  # its own work items are made by its first product
                fv.logreg_eval(A, label, w, storage=s)
                assert A.device_bytes == used, s
        assert A.panel_info()[2] > 0 and A.head_info()[0] == 64
        A.close()
