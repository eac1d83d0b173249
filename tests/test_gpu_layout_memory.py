"""Device memory of the row panels and the forward head: the streamed records hold a value and a 2-byte slot per entry
(as the storage keeps the value: 2, 4 or 4 + 2 bytes), and nothing else grows with the entries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dense(m, n):
    rng = np.random.default_rng(0)
    off = np.arange(m + 1, dtype=np.int32) * n
    idx = np.tile(np.arange(n, dtype=np.int32), m)
    val = (rng.standard_normal(m * n).astype(np.float32).view(np.uint32) & 0xFFFF0000).view(np.float32)
    return off, idx, val


@pytest.mark.parametrize("storage,entry", [("bf16", 4), ("f32", 6), ("split", 8)])
@pytest.mark.parametrize("layout", ["panels", "head"])
def test_bytes_per_entry(storage, entry, layout):
    import frovedis_gb300 as fv
    m, n = 20_000, 160
    off, idx, val = _dense(m, n)
    v = {"bf16": (val.view(np.uint32) >> 16).astype(np.uint16), "f32": val, "split": val.astype(np.float64)}[storage]
    label = np.where(np.arange(m) % 2 == 0, 1.0, -1.0)
    w = np.linspace(-1.0, 1.0, n)
    used, out = [], []
    with fv.Context(0) as ctx:
        for on in (False, True):
            A = ctx.matrix(m, n, off, idx, v)
            A.set_panels(10_000 if on and layout == "panels" else 0, 1.0)
            A.set_head(n if on and layout == "head" else 0)
            out.append(fv.logreg_eval(A, label, w, storage=storage))
            used.append(A.device_bytes)
            A.close()
    rows = 2 * n if layout == "panels" else m
    per_row = 64  # offsets, sums and segment places of a row of the layout
    assert used[1] - used[0] <= 1.1 * entry * m * n + per_row * rows + (1 << 20)
    assert np.allclose(out[0][0], out[1][0], rtol=1e-4, atol=1e-2 * np.abs(out[0][0]).max())
