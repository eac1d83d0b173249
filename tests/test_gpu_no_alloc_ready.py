"""Which matrices the product without allocations takes: any that has work items, in every storage it holds values of,
whatever call made them first.  Tolerance: as the other products', FP64 1e-12 and FP32 2e-5 of a row's sum of
magnitudes."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,first", [("f32", "add_split"), ("f32", "eval_split"), ("f64", "eval_f32"),
                                           ("f32", "prepare"), ("f64", "prepare")])
def test_accepted(storage, first):
    torch = pytest.importorskip("torch")
    import frovedis_gb300 as fv
    from frovedis_gb300 import datagen
    off, idx, val, label = datagen.generate(datagen.Spec(m=3000, n=900, lam=15.0, seed=6))
    a = oracle.CRS(3000, 900, off, idx, val)
    w = np.linspace(-1.0, 1.0, a.n)
    with fv.Context(0) as ctx:
        A = ctx.matrix(a.m, a.n, off, idx, val)
        if first != "eval_f32":
            A.prepare("CRS", transpose=False)
        if first == "add_split":
            A.add_storage("split")
        elif first == "eval_split":
            fv.logreg_eval(A, label, w, storage="split")
        elif first == "eval_f32":
            fv.logreg_eval(A, label, w, storage="f32")
        else:
            A.add_storage(storage)
        vec = "f64" if storage == "f64" else "f32"
        x = torch.from_numpy(w).cuda().to(torch.float64 if vec == "f64" else torch.float32)
        y = torch.full((a.m,), float("nan"), dtype=x.dtype, device="cuda")
        torch.cuda.synchronize()
        rc = ctx.L.fvg_spmv_no_alloc(ctx.h, A.h, fv.DTYPES[storage], fv.DTYPES[vec], ctypes.c_void_p(x.data_ptr()),
                                     ctypes.c_void_p(y.data_ptr()))
        assert rc == 0, ctx.L.fvg_ctx_last_error(ctx.h)
        ctx.synchronize()
        want = oracle.spmv(a, x.cpu().numpy().astype(np.float64))
        mag = oracle.spmv(oracle.CRS(a.m, a.n, off, idx, np.abs(val)), np.abs(w))
        tol = 1e-12 if storage == "f64" else 2e-5
        assert np.all(np.abs(y.cpu().numpy() - want) <= tol * (mag + 1e-30))
        A.close()
