"""The work that programs give to this library, one pass at a time.

A case names an operation of the public Python interface and the shape of its
sparse matrix:

  product       y = A x or y = A^T x on device vectors (operator*, trans_mv)
  spmm          Y = A X with a dense block of k columns on the device
  predict       class-1 probabilities of a trained model for a matrix of samples
  eval          one loss / gradient evaluation of a linear model
  lbfgs         a whole L-BFGS training of one model
  sgd           a whole minibatch SGD training of one model
  path          a regularisation path: k models trained together by L-BFGS
  multinomial   a whole softmax L-BFGS training

Matrices follow the benchmark configurations' distributions: 1 + Poisson row
lengths with Zipf column ids (click-through and text data) or power-law row
lengths with uniform column ids (graphs), drawn on the GPU from the seed.
"""
import math

import numpy as np
import torch

import frovedis_gb300 as fv

DEV = "cuda"
LOGISTIC, SQUARED, HINGE = "logistic", "linear", "hinge"

_context = None


def _ctx():
    """The program's one context."""
    global _context
    if _context is None:
        _context = fv.Context(0)
    return _context


# ------------------------------------------------------------------- cases
def listed():
    return [
        # a product of a model-sized matrix inside somebody's own loop: the call itself is what counts
        dict(name="product small f64", op="product", trans=False, fmt="CRS", storage="f64", m=3000, n=400, avg=13.0,
             rows="poisson", zipf=1.1),
        # graph-like matrix, the default format and precision, forward
        dict(name="product 2M crs f64", op="product", trans=False, fmt="CRS", storage="f64", m=2_000_000,
             n=2_000_000, avg=40.0, rows="zipf", zipf=0.0),
        # the same matrix transposed in the format made for skewed row lengths, single precision
        dict(name="trans 2M jds f32", op="product", trans=True, fmt="JDS", storage="f32", m=2_000_000, n=2_000_000,
             avg=40.0, rows="zipf", zipf=0.0),
        # gradient-like product over a click-through matrix kept in 16 bits
        dict(name="trans 2M bf16", op="product", trans=True, fmt="CRS", storage="bf16", m=2_000_000, n=200_000,
             avg=60.0, rows="poisson", zipf=1.1),
        # scores of 64 models for one data set of the regularisation-path workload
        dict(name="spmm 64 f32", op="spmm", storage="f32", m=300_000, n=500_000, avg=50.0, rows="poisson", zipf=1.2,
             k=64),
        # scoring a batch of samples with a trained model, host in, host out
        dict(name="predict 100k", op="predict", m=100_000, n=20_000, avg=40.0, rows="poisson", zipf=1.1),
        # one weighted SVM loss / gradient evaluation, for a caller with an optimiser of its own
        dict(name="eval hinge 1M f64", op="eval", loss=HINGE, storage="f64", m=1_000_000, n=100_000, avg=60.0,
             rows="poisson", zipf=1.1, weighted=True),
        # the sample program's training: 100,000 x 20,000, 20 iterations, double precision
        dict(name="lbfgs 100k f64", op="lbfgs", storage="f64", m=100_000, n=20_000, avg=40.0, rows="poisson",
             zipf=1.1, iters=20, reg=1e-3, intercept=False),
        # training at scale on split values, the arm the benchmark leads with
        dict(name="lbfgs 10M split", op="lbfgs", storage="split", m=10_000_000, n=1_000_000, avg=60.0,
             rows="poisson", zipf=1.1, iters=10, reg=1e-4, intercept=False),
        # the other solver, in minibatches
        dict(name="sgd 100k f64", op="sgd", storage="f64", m=100_000, n=20_000, avg=40.0, rows="poisson", zipf=1.1,
             iters=20, reg=1e-3, fraction=0.25),
        # 64 regularisation values on one data set, 16-bit values
        dict(name="path 64 bf16", op="path", storage="bf16", m=200_000, n=20_000, avg=50.0, rows="poisson", zipf=1.2,
             iters=5, k=64),
        # softmax training, 16-bit values
        dict(name="multinomial 32 bf16", op="multinomial", storage="bf16", m=1_000_000, n=50_000, avg=100.0,
             rows="poisson", zipf=1.1, iters=3, k=32, reg=1e-4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _matrix(rng, m_lo, m_hi, nnz_max, n_hi=2_000_000):
    """A drawn matrix shape: any row count of the range, a width from a fraction of it up to as wide."""
    m = _log_int(rng, m_lo, m_hi)
    n = max(50, min(n_hi, _log_int(rng, m / 20.0, m)))
    avg = round(rng.uniform(4.0, 80.0), 1)
    avg = round(max(2.0, min(avg, nnz_max / m, n / 4.0)), 1)
    if rng.random() < 0.25:
        return dict(m=m, n=n, avg=avg, rows="zipf", zipf=0.0)
    return dict(m=m, n=n, avg=avg, rows="poisson", zipf=rng.choice([1.05, 1.1, 1.2]))


def draw(rng):
    op = rng.choice(["product", "product", "product", "spmm", "predict", "eval", "lbfgs", "lbfgs", "sgd", "path",
                     "multinomial"])
    if op == "product":
        c = dict(op=op, trans=rng.random() < 0.5, **_matrix(rng, 1000, 4_000_000, 200e6))
        c["storage"] = rng.choice(["f64", "f64", "f32", "bf16", "split"])
        fmts = ["CRS", "CRS", "JDS", "HYBRID"] + (["ELL"] if c["rows"] == "poisson" else [])
        c["fmt"] = "CRS" if c["storage"] == "split" else rng.choice(fmts)
        return c
    if op == "spmm":
        return dict(op=op, storage=rng.choice(["f64", "f32", "f32", "bf16"]), k=rng.randint(1, 128),
                    **_matrix(rng, 5000, 400_000, 20e6))
    if op == "predict":
        return dict(op=op, **_matrix(rng, 1000, 1_000_000, 50e6, 500_000))
    if op == "eval":
        return dict(op=op, loss=rng.choice([LOGISTIC, SQUARED, HINGE]), storage=rng.choice(["f64", "split"]),
                    weighted=rng.random() < 0.5, **_matrix(rng, 5000, 3_000_000, 150e6, 500_000))
    if op == "lbfgs":
        split = rng.random() < 0.5
        return dict(op=op, storage="split" if split else "f64", iters=rng.randint(5, 10 if split else 20),
                    reg=rng.choice([1e-4, 1e-3]), intercept=rng.random() < 0.3,
                    **_matrix(rng, 5000, 4_000_000 if split else 400_000, 240e6 if split else 20e6, 400_000))
    if op == "sgd":
        return dict(op=op, storage="f64", iters=rng.randint(5, 20), reg=1e-3,
                    fraction=rng.choice([0.1, 0.25, 0.5, 1.0]), **_matrix(rng, 5000, 300_000, 15e6, 100_000))
    if op == "path":
        return dict(op=op, storage=rng.choice(["f64", "f32", "bf16"]), iters=rng.randint(2, 5), k=rng.randint(2, 64),
                    **_matrix(rng, 5000, 200_000, 10e6, 40_000))
    return dict(op=op, storage=rng.choice(["f32", "bf16"]), iters=rng.randint(2, 3), k=rng.randint(3, 128), reg=1e-4,
                **_matrix(rng, 5000, 200_000, 10e6, 20_000))


# ------------------------------------------------------------------ inputs
def _gen(seed, stream):
    return torch.Generator(device=DEV).manual_seed(1_000_003 * int(seed) + stream)


def _zipf_cdf(n, s):
    """Summed on the host, in one fixed order: the same table for the same case every time."""
    c = np.cumsum(np.arange(1, n + 1, dtype=np.float64) ** -s)
    return torch.from_numpy(c / c[-1]).to(DEV)


def _row_lengths(case, seed):
    m, n, avg = case["m"], case["n"], case["avg"]
    g = _gen(seed, 1)
    if case["rows"] == "poisson":
        # a column id drawn twice in a row counts once: draw some more of the frequent ones
        extra = 1.35 if case["zipf"] > 0 and n > 1000 else 1.0
        lens = 1 + torch.poisson(torch.full((m,), max(avg - 1.0, 0.0) * extra, device=DEV), generator=g).long()
    else:
        cap = min(20_000, n)
        u = torch.rand(m, device=DEV, dtype=torch.float64, generator=g)
        raw = (torch.searchsorted(_zipf_cdf(cap, 1.3), u) + 1).clamp_(max=cap).double()
        raw *= avg * m / raw.sum()
        lens = torch.floor(raw + torch.rand(m, device=DEV, dtype=torch.float64, generator=g)).long().clamp_(max=cap)
    return lens.clamp_(max=n)


def _crs(case, seed):
    """off (int32), idx (int32), val (float64) of the case's matrix on the GPU: distinct ascending ids in each row."""
    m, n = case["m"], case["n"]
    lens = _row_lengths(case, seed)
    starts = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(lens, 0, out=starts[1:])
    total = int(starts[-1])
    cdf = _zipf_cdf(n, case["zipf"]) if case["zipf"] > 0 else None
    g = _gen(seed, 2)
    idx = torch.empty(total, dtype=torch.int32, device=DEV)
    counts = torch.zeros(m, dtype=torch.int64, device=DEV)
    step = 1 << 26  # draws made at a time
    bounds = torch.searchsorted(starts, torch.arange(0, total, step, device=DEV), right=True).sub_(1).tolist()
    cuts = sorted(set(bounds + [m]))
    kept = 0
    for r0, r1 in zip(cuts[:-1], cuts[1:]):
        ln = lens[r0:r1]
        key = torch.repeat_interleave(torch.arange(r1 - r0, device=DEV), ln)
        u = torch.rand(key.numel(), device=DEV, dtype=torch.float64, generator=g)
        col = (torch.searchsorted(cdf, u) if cdf is not None else (u * n).long()).clamp_(max=n - 1)
        key = key.mul_(n).add_(col)
        del u, col
        key = torch.unique_consecutive(torch.sort(key).values)
        idx[kept:kept + key.numel()] = key.remainder(n).int()
        counts[r0:r1] = torch.bincount(key.div_(n, rounding_mode="floor"), minlength=r1 - r0)
        kept += key.numel()
        del key
    off = torch.zeros(m + 1, dtype=torch.int32, device=DEV)
    off[1:] = torch.cumsum(counts, 0).int()
    idx = idx[:kept].clone() if kept < total else idx
    val = torch.empty(kept, dtype=torch.float64, device=DEV)
    val.normal_(generator=_gen(seed, 3))
    if case["rows"] == "poisson":
        val.mul_(0.5).exp_()  # lognormal counts, as the benchmark's
    return off, idx, val


def _stored(case, val):
    """The values as the program holds them before the call: narrow ones are uploaded narrow."""
    return {"f32": val.float, "bf16": val.bfloat16}.get(case.get("storage", "f64"), lambda: val)()


def _as_matrix(case, off, idx, val):
    dtype = {torch.float64: fv.F64, torch.float32: fv.F32, torch.bfloat16: fv.BF16}[val.dtype]
    torch.cuda.synchronize()
    return _ctx().matrix(case["m"], case["n"], off.data_ptr(), idx.data_ptr(), (val.data_ptr(), dtype), on_device=True)


def _times_rows(off, idx, val, x):
    """A x in double precision for making labels (x a vector)."""
    m = off.numel() - 1
    out = torch.zeros(m, dtype=torch.float64, device=DEV)
    step = 1 << 27
    row = torch.repeat_interleave(torch.arange(m, device=DEV, dtype=torch.int32), (off[1:] - off[:-1]).long())
    for a in range(0, idx.numel(), step):
        s = slice(a, a + step)
        out.index_add_(0, row[s], val[s] * x[idx[s]])
    return out


def _model(case, seed, stream, k=1):
    w = torch.empty(k, case["n"], dtype=torch.float64, device=DEV)
    return w.normal_(generator=_gen(seed, stream)).mul_(1.0 / math.sqrt(max(case["avg"], 1.0)))


def _labels(case, seed, off, idx, val):
    """+-1 from a hidden model's probabilities, or real targets for the squared loss; class ids for a softmax."""
    g = _gen(seed, 5)
    if case["op"] == "multinomial":
        few = min(case["k"], 8)  # the classes of a sample follow a few hidden scores
        scores = torch.stack([_times_rows(off, idx, val, w) for w in _model(case, seed, 4, few)], 1)
        top = torch.argmax(scores + torch.rand(scores.shape, device=DEV, dtype=torch.float64, generator=g), 1)
        other = torch.randint(0, case["k"], top.shape, device=DEV, generator=g)
        return torch.where(torch.rand(top.shape, device=DEV, generator=g) < 0.7, top, other).double()
    z = _times_rows(off, idx, val, _model(case, seed, 4)[0])
    if case.get("loss") == SQUARED:
        return z + 0.1 * torch.empty_like(z).normal_(generator=g)
    return torch.where(torch.rand(z.shape, device=DEV, dtype=torch.float64, generator=g) < torch.sigmoid(z), 1.0, -1.0)


def _pinned(t):
    """A loader's staging buffer: the array in page-locked host memory."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _path_values(case):
    return np.logspace(-6, 0, case["k"])


def _vec(case):
    return ("f64", torch.float64) if case["storage"] in ("f64", "split") else ("f32", torch.float32)


def _arrays(case, seed):
    """Everything a pass reads: the matrix on the GPU and what goes with it (also what exact() starts from)."""
    off, idx, val = _crs(case, seed)
    d = dict(off=off, idx=idx)
    op = case["op"]
    if op == "product":
        d["x"] = torch.empty(case["m" if case["trans"] else "n"], dtype=torch.float64, device=DEV).normal_(
            generator=_gen(seed, 6)).to(_vec(case)[1])
    elif op == "spmm":
        d["x"] = torch.empty(case["n"], case["k"], dtype=torch.float64, device=DEV).normal_(
            generator=_gen(seed, 6)).to(_vec(case)[1])
    elif op == "predict":
        d["w"] = _model(case, seed, 6)[0]
    else:
        d["label"] = _labels(case, seed, off, idx, val)
        if op == "eval":
            d["w"] = _model(case, seed, 6)[0]
            d["sw"] = None
            if case["weighted"]:
                d["sw"] = 0.5 + torch.rand(case["m"], device=DEV, dtype=torch.float64, generator=_gen(seed, 7))
    d["val"] = _stored(case, val)
    return d


def prepare(case, seed):
    op = case["op"]
    d = _arrays(case, seed)
    A = _as_matrix(case, d["off"], d["idx"], d["val"])
    s = dict(case=case, A=A)
    storage = case.get("storage", "f64")
    if storage == "split":
        A.add_storage("split")
    A.prepare(case.get("fmt", "CRS"), transpose=op not in ("spmm", "predict") and case.get("trans", True))
    if op in ("product", "spmm"):
        s["x"] = d["x"]
        shape = (case["m"], case["k"]) if op == "spmm" else (case["n" if case["trans"] else "m"],)
        s["y"] = torch.empty(shape, dtype=d["x"].dtype, device=DEV)
    elif op == "predict":
        s["w"] = d["w"].cpu().numpy()
    else:
        s["label"] = _pinned(d["label"])
        if op == "eval":
            s["w"] = d["w"].cpu().numpy()
            s["sw"] = None if d["sw"] is None else _pinned(d["sw"])
        elif op != "multinomial":
            s["w0"] = np.zeros(case["n"])
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------- run
def _narrow(case, w):
    """A trained model as a program keeps it: values of 32 bits or fewer give a model of 32 bits."""
    return w if case["storage"] in ("f64", "split") else w.astype(np.float32)


def run(s):
    case, A = s["case"], s["A"]
    op = case["op"]
    if op == "product":
        call = A.trans_mv_device if case["trans"] else A.spmv_device
        call(s["x"].data_ptr(), s["y"].data_ptr(), fmt=case["fmt"], storage=case["storage"], vec=_vec(case)[0])
        return s["y"]
    if op == "spmm":
        A.spmm_device(s["x"].data_ptr(), case["k"], s["y"].data_ptr(), storage=case["storage"], vec=_vec(case)[0])
        return s["y"]
    if op == "predict":
        return fv.predict_probability(A, s["w"], 0.25)
    if op == "eval":
        g, loss = fv.glm_eval(A, s["label"], s["w"], b=0.25, intercept=True, sample_weight=s["sw"],
                              storage=case["storage"], loss=case["loss"])
        return [g, loss]
    if op == "lbfgs":
        r = fv.logreg_lbfgs(A, s["label"], w0=s["w0"], b0=0.0, num_iter=case["iters"], reg_type="L2",
                            reg_param=case["reg"], intercept=case["intercept"], storage=case["storage"])
        return [r["w"], r["b"], r["loss"], r["n_iter"]]
    if op == "sgd":
        r = fv.logreg_sgd(A, s["label"], w0=s["w0"], num_iter=case["iters"], alpha=4.0 / case["m"], reg_type="L2",
                          reg_param=case["reg"], mini_batch_fraction=case["fraction"], convergence_tol=0.0,
                          storage=case["storage"])
        return [r["w"], r["loss"], r["n_iter"]]
    if op == "path":
        r = fv.logreg_lbfgs_batched(A, s["label"], _path_values(case), w0=s["w0"], num_iter=case["iters"],
                                    reg_type="L2", storage=case["storage"])
        return [_narrow(case, r["w"]), _narrow(case, r["loss"]), r["n_iter"]]
    r = fv.multinomial_lbfgs(A, s["label"], case["k"], num_iter=case["iters"], reg_type="L2", reg_param=case["reg"],
                             storage=case["storage"])
    return [_narrow(case, r["W"]), _narrow(case, np.float64(r["loss"])), r["n_iter"]]


# -------------------------------------------------------------------- work
def work(case):
    """Each input read once and each output written once: a matrix entry is its value and a 4-byte id."""
    m, n, op = case["m"], case["n"], case["op"]
    z = m * case["avg"]
    sv = {"f64": 8, "f32": 4, "bf16": 2, "split": 6}[case.get("storage", "f64")]
    sx = 8 if case.get("storage", "f64") in ("f64", "split") else 4
    one = z * (sv + 4) + 4 * m
    if op == "product":
        return {"bytes": one + (m + n) * sx, "flops": 2 * z}
    if op == "spmm":
        return {"bytes": one + (m + n) * sx * case["k"], "flops": 2 * z * case["k"]}
    if op == "predict":
        return {"bytes": one + 8 * (m + n), "flops": 2 * z}
    if op == "eval":
        return {"bytes": one + 8 * m * (2 if case["weighted"] else 1) + 16 * n, "flops": 4 * z}
    # a training reads the matrix for A w and again for A^T r in every evaluation (one more than iterations)
    k = case.get("k", 1)
    evals = case["iters"] + (0 if op == "sgd" else 1)
    return {"bytes": evals * (2 * one + 8 * m + 16 * n * k), "flops": evals * 4 * z * k}


# ------------------------------------------------------------------- exact
class _Csr64:
    """A and A^T in double precision for torch's own sparse products."""

    def __init__(self, case, d, trans=True):
        m, n = case["m"], case["n"]
        off, idx, val = d["off"], d["idx"], d["val"].double()
        self.a = torch.sparse_csr_tensor(off, idx, val, (m, n))
        if trans:
            perm = torch.sort(idx, stable=True).indices
            row = torch.repeat_interleave(torch.arange(m, device=DEV, dtype=torch.int32), (off[1:] - off[:-1]).long())
            toff = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
            toff[1:] = torch.cumsum(torch.bincount(idx, minlength=n), 0).int()
            self.t = torch.sparse_csr_tensor(toff, row[perm], val[perm], (n, m))


def _dloss(kind, z, y):
    """Loss sum and derivative by the prediction z of each sample."""
    if kind == SQUARED:
        return 0.5 * ((z - y) ** 2).sum(), z - y
    t = y * z
    if kind == HINGE:
        return torch.clamp(1.0 - t, min=0.0).sum(), torch.where(t <= 1.0, -y, torch.zeros_like(y))
    e = torch.exp(-t.abs())
    return (torch.clamp(-t, min=0.0) + torch.log1p(e)).sum(), -y * torch.where(t > 0, e, torch.ones_like(e)) / (1.0 + e)


def _minimise(f, x, bias, iters, reg):
    """The L-BFGS of the library's interface on x (weights, then the intercept) in plain torch: history 10, at most
    ten step lengths a tenth of the one before, L2 shrinkage after each step, a stop at a gradient rms of 1e-3."""
    pairs = []
    x = torch.cat([x, torch.tensor([bias], dtype=torch.float64, device=DEV)])
    loss, g = f(x)
    it = 1
    while it <= iters:
        if not pairs:
            c = float(g.norm())
            d = -(-(c if c <= 1 else 1 / c) * 0.1 * g)
        else:
            q, al = g.clone(), []
            for s, y, rho in reversed(pairs):
                al.append(rho * torch.dot(s, q))
                q -= al[-1] * y
            s, y, rho = pairs[-1]
            yy = torch.dot(y, y)
            z = q * ((1.0 / rho) / (yy if float(yy) else 1.0))
            for (s, y, rho), a in zip(pairs, reversed(al)):
                z += (a - rho * torch.dot(y, z)) * s
            d = -z
        if float(torch.dot(g, d)) > 0:
            d = -d
        size = float(d.norm())
        eta = 1.0 if size <= 1e20 else 1e20 / size
        for _ in range(10):
            nx = x + eta * d
            nx[:-1] *= max(0.0, 1.0 - reg * eta)
            nloss, ng = f(nx)
            if float(nloss) - float(loss) < 1e-4:
                break
            eta /= 10.0
        s, y = nx - x, ng - g
        y = torch.where(y.abs() < 1e-10, torch.zeros_like(y), y)
        sy = torch.dot(s, y)
        pairs = (pairs + [(s, y, 1.0 / (sy if float(sy) else torch.ones_like(sy)))])[-10:]
        x, g, loss = nx, ng, nloss
        if float(g.norm()) / math.sqrt(g.numel()) <= 1e-3:
            break
        it += 1
    return x[:-1], float(x[-1]), float(loss), min(it, iters)


def _binary(A, d, kind, weight, intercept):
    def f(x):
        z = A.a @ x[:-1]
        if intercept:
            z = z + x[-1]
        loss, r = _dloss(kind, z, d["label"])
        if weight is not None:
            r = r * weight
        b = r.sum().reshape(1) if intercept else torch.zeros(1, dtype=torch.float64, device=DEV)
        return loss, torch.cat([A.t @ r, b])
    return f


def exact(case, seed):
    op, n = case["op"], case["n"]
    d = _arrays(case, seed)
    if op in ("product", "spmm"):
        trans = case.get("trans", False)
        A = _Csr64(case, d, trans)
        return (A.t if trans else A.a) @ d["x"].double()
    if op == "predict":
        return torch.sigmoid(_Csr64(case, d, False).a @ d["w"] + 0.25)
    A = _Csr64(case, d)
    zero = torch.zeros(n, dtype=torch.float64, device=DEV)
    if op == "eval":
        loss, g = _binary(A, d, case["loss"], d["sw"], True)(torch.cat([d["w"], torch.full_like(d["w"][:1], 0.25)]))
        return [g, float(loss)]
    if op == "lbfgs":
        f = _binary(A, d, LOGISTIC, None, case["intercept"])
        w, b, loss, _ = _minimise(f, zero, 0.0, case["iters"], case["reg"])
        return [w, b if case["intercept"] else 0.0, loss, None]
    if op == "path":
        f = _binary(A, d, LOGISTIC, None, False)
        got = [_minimise(f, zero, 0.0, case["iters"], float(lam)) for lam in _path_values(case)]
        return [torch.stack([w for w, _, _, _ in got]), torch.tensor([x for _, _, x, _ in got], dtype=torch.float64),
                None]
    if op == "sgd":
        return _exact_sgd(case, d)
    k = case["k"]
    hot = torch.nn.functional.one_hot(d["label"].long(), k).double()

    def f(x):
        z = A.a @ x[:-1].reshape(n, k)
        logp = torch.log_softmax(z, 1)
        return -(logp * hot).sum(), torch.cat([(A.t @ (logp.exp() - hot)).reshape(-1), x[-1:] * 0.0])

    w, _, loss, _ = _minimise(f, torch.zeros(n * k, dtype=torch.float64, device=DEV), 0.0, case["iters"], case["reg"])
    return [w.reshape(n, k), loss, None]


def _exact_sgd(case, d):
    m, n = case["m"], case["n"]
    size = min(m, -(-math.ceil(m * case["fraction"]) // 1024) * 1024)
    batches = []
    for r0 in range(0, m, size):
        r1 = min(m, r0 + size)
        a, b = int(d["off"][r0]), int(d["off"][r1])
        part = dict(off=(d["off"][r0:r1 + 1] - a).contiguous(), idx=d["idx"][a:b].contiguous(), val=d["val"][a:b])
        batches.append((_Csr64(dict(m=r1 - r0, n=n), part), d["label"][r0:r1]))
    w = torch.zeros(n, dtype=torch.float64, device=DEV)
    loss = 0.0
    for i in range(1, case["iters"] + 1):
        step = 4.0 / m / math.sqrt(i)
        loss = 0.0
        for A, y in batches:
            part, r = _dloss(LOGISTIC, A.a @ w, y)
            w = w - step * (A.t @ r)
            loss += float(part)
        w = w * max(0.0, 1.0 - case["reg"] * step)
    return [w, loss, None]
