"""The work that users of fastpls_b200 have it do, as measured cases.

Each case is one call (or one short chain of calls) of the public binding
``fastpls_b200._lib`` on seeded synthetic data.  The kinds:

  simpls  fast SIMPLS regression, FP64: fit, then prediction of held-out rows
  plslda  PLSSVD + LDA classification in one fused call, FP32 or FP64 features
  dcv     double cross-validation of a SIMPLS classifier on a registered matrix
  cknn    label-aware PLSSVD + candidate kNN on registered FP32 features
  opls    OPLS filter, Gaussian response compression, SIMPLS, filtered test
          prediction and decoding
  topk    top-k class prediction of new rows under a kept model (serving)

Matrices are column-major in device memory, as a program that keeps its data on
the GPU passes them; label vectors, fold ids and small model fields are host
arrays, as the binding takes them.
"""
import math

import numpy as np
import torch

from fastpls_b200 import _lib as lib
from fastpls_b200.folds import double_cv_folds


def listed():
    return [
        # a regression of a few hundred samples (400 x 2000, five responses):
        # the everyday small call, bound by launches and latency
        dict(name="simpls_small", kind="simpls", n=400, p=2000, m=5, k=10, n_test=100),
        # a metabolomics-sized classifier (773 x 375 in all, 22 classes), three
        # component counts: the smallest call, as model selection repeats it
        dict(name="plslda_small", kind="plslda", n=618, p=375, classes=22, k=20, slices=3, n_test=155,
             dtype="float64", precision="fp64"),
        # the tall regression sweep: 50000 x 1000, 100 responses, 5 components
        dict(name="simpls_tall", kind="simpls", n=50000, p=1000, m=100, k=5, n_test=10000),
        # image features, 100 classes, two component counts, FP64 arithmetic
        dict(name="plslda_features", kind="plslda", n=50000, p=768, classes=100, k=50, slices=2, n_test=10000,
             dtype="float32", precision="fp64"),
        # wide PLS-DA, split-precision products
        dict(name="plslda_wide", kind="plslda", n=20000, p=5000, classes=100, k=50, slices=1, n_test=5000,
             dtype="float32", precision="bf16x3"),
        # the double-CV grid of 1500 fits on omics data, mixed precision
        dict(name="dcv_omics_bf16x3", kind="dcv", n=3000, p=20000, classes=4, outer=10, inner=5, k=30,
             precision="bf16x3"),
        # the same kind of grid at half the samples in the INT8 form (the one
        # whose scores stay within 1e-5 of FP64)
        dict(name="dcv_omics_int8", kind="dcv", n=1500, p=8000, classes=4, outer=10, inner=5, k=30,
             precision="int8"),
        # a small study in plain FP64, odd sizes, uneven folds
        dict(name="dcv_ragged_fp64", kind="dcv", n=777, p=4099, classes=3, outer=7, inner=4, k=15,
             precision="fp64"),
        # more samples than features: the predictor-space engine
        dict(name="dcv_tall_fp64", kind="dcv", n=5000, p=501, classes=5, outer=5, inner=5, k=20,
             precision="fp64"),
        # 1.2 million rows, 1000 skewed classes: the large-scale classifier
        dict(name="cknn_large", kind="cknn", n=1200000, p=768, classes=1000, k=100, n_test=50000),
        # multi-response chemometrics with an orthogonal filter
        dict(name="opls_response", kind="opls", n=20000, p=8000, q=1000, dim=100, north=2, k=50, n_test=4000,
             precision="bf16x6"),
        # serving: 20000 new rows against a kept 1000-class model
        dict(name="predict_topk", kind="topk", n=20000, p=768, classes=1000, k=100, top=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["simpls", "simpls", "plslda", "plslda", "dcv", "dcv", "cknn", "opls", "topk"])
    if kind == "simpls":
        n = _log(rng, 150, 50000)
        p = min(_log(rng, 50, 4000), 50_000_000 // n)
        return dict(kind=kind, n=n, p=p, m=_log(rng, 2, 100), k=rng.randint(2, 10), n_test=_log(rng, 20, 10000))
    if kind == "plslda":
        n = _log(rng, 400, 50000)
        p = min(_log(rng, 100, 5000), 100_000_000 // n)
        classes = _log(rng, 4, min(100, n // 12))
        return dict(kind=kind, n=n, p=p, classes=classes, k=rng.randint(2, min(50, classes - 2)),
                    slices=rng.randint(1, 3), n_test=_log(rng, 20, 10000),
                    dtype=rng.choice(["float32", "float64"]), precision=rng.choice(["fp64", "bf16x3"]))
    if kind == "dcv":
        if rng.random() < 0.35:   # more samples than half the features
            n = _log(rng, 400, 5000)
            p = _log(rng, 100, min(1500, 2 * n - 1))
            k, prec = rng.randint(4, 20), rng.choice(["fp64", "bf16x3"])
        else:
            n = _log(rng, 200, 3000)
            p = _log(rng, max(2 * n, 600), 20000)
            k, prec = rng.randint(5, 30), rng.choice(["fp64", "bf16x3", "int8"])
        return dict(kind=kind, n=n, p=p, classes=rng.randint(2, 5), outer=rng.randint(3, 10),
                    inner=rng.randint(3, 5), k=k, precision=prec)
    if kind == "cknn":
        classes = _log(rng, 50, 1000)
        p = _log(rng, 64, 768)
        return dict(kind=kind, n=_log(rng, 20000, 1200000), p=p, classes=classes,
                    k=rng.randint(10, min(100, p // 2, classes // 2)), n_test=_log(rng, 500, 50000))
    if kind == "opls":
        return dict(kind=kind, n=_log(rng, 1000, 20000), p=_log(rng, 500, 8000), q=_log(rng, 120, 1000),
                    dim=rng.randint(40, 100), north=rng.randint(1, 3), k=rng.randint(5, 50),
                    n_test=_log(rng, 100, 4000), precision=rng.choice(["fp64", "bf16x6"]))
    return dict(kind=kind, n=_log(rng, 50, 20000), p=_log(rng, 100, 4000), classes=_log(rng, 10, 1000),
                k=rng.randint(5, 100), top=rng.randint(1, 10))


# ------------------------------------------------------------------ inputs ---
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _randn(g, rows, cols, dtype=torch.float64):
    """A rows x cols column-major normal matrix."""
    return torch.randn(cols, rows, generator=g, device="cuda", dtype=dtype).T


def _colmajor(a):
    return a.T.contiguous().T


def _lowrank_x(g, n, p, rank, scale, noise):
    """A latent signal with geometrically falling strengths plus noise."""
    rank = min(rank, n, p)
    u = _randn(g, n, rank) / math.sqrt(n)
    v = _randn(g, p, rank) / math.sqrt(p)
    s = scale * 0.8 ** torch.arange(rank, device="cuda", dtype=torch.float64)
    x = torch.matmul(v, (u * s).T).T          # column-major n x p
    return x.add_(_randn(g, n, p), alpha=noise)


def _labels(g, n, classes, weights=None):
    """0-based labels, every class present."""
    if weights is None:
        y = torch.arange(n, device="cuda") % classes
    else:
        w = torch.as_tensor(weights, dtype=torch.float64, device="cuda")
        y = torch.multinomial(w, n, replacement=True, generator=g)
        y[:classes] = torch.arange(classes, device="cuda")
    return y[torch.randperm(n, generator=g, device="cuda")]


class _Registered:
    """A registered (library-owned) matrix that is released with its owner."""

    def __init__(self, x):
        self.m = lib.x_alloc(x.shape[0], x.shape[1], f32=x.dtype == torch.float32)
        torch.as_tensor(self.m, device="cuda").copy_(x)
        torch.cuda.synchronize()
        self.handle = self.m.handle

    def __del__(self):
        try:
            lib.x_free(self.handle)
        except Exception:   # the library is already gone at interpreter exit
            pass


def _inputs(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = {}
    if kind == "simpls":
        n, nt = case["n"], case["n_test"]
        x = _lowrank_x(g, n + nt, case["p"], 20, 10.0 * math.sqrt(case["p"]), 1.0)
        b = _randn(g, case["p"], case["m"]) / math.sqrt(case["p"])
        y = x @ b + 0.5 * _randn(g, n + nt, case["m"])
        s["x"], s["y"], s["xt"] = _colmajor(x[:n]), _colmajor(y[:n]), _colmajor(x[n:])
    elif kind == "plslda":
        n, nt, c = case["n"], case["n_test"], case["classes"]
        dt = torch.float32 if case["dtype"] == "float32" else torch.float64
        mu = 0.5 * _randn(g, c, case["p"], dt)
        lab = torch.cat([_labels(g, n, c), torch.randint(c, (nt,), generator=g, device="cuda")])
        x = _randn(g, n + nt, case["p"], dt).add_(_colmajor(mu[lab]))
        s["x"], s["xt"] = _colmajor(x[:n]), _colmajor(x[n:])
        s["lab"] = lab[:n]
        s["y"] = _colmajor((lab[:n, None] == torch.arange(c, device="cuda")[None, :]).double())
    elif kind == "dcv":
        n, p, c = case["n"], case["p"], case["classes"]
        w = np.arange(c, 0, -1, dtype=np.float64)
        lab = _labels(g, n, c, w / w.sum())
        x = torch.log1p(torch.exp(_randn(g, n, p, torch.float32)))
        inf = torch.randperm(p, generator=g, device="cuda")[:max(10, min(50, p // 4))]
        x[:, inf] += (0.5 * x[:, inf].std(dim=0))[None, :] * lab[:, None].float()
        x -= x.mean(dim=0, keepdim=True)
        sizes = torch.randint(1, 6, (n,), generator=g, device="cuda").cpu().numpy()
        groups = np.repeat(np.arange(1, n + 1), sizes)[:n].astype(np.int32)
        s["x"] = _colmajor(x)
        s["y"] = (lab.cpu().numpy() + 1).astype(np.int32)
        s["outer"], s["inner"] = double_cv_folds(s["y"], groups, case["outer"], case["inner"], seed=int(seed))
    elif kind == "cknn":
        n, nt, p, c = case["n"], case["n_test"], case["p"], case["classes"]
        proto = _randn(g, c, p, torch.float32)
        proto = proto / proto.norm(dim=1, keepdim=True)
        zipf = 1.0 / np.arange(1, c + 1) ** 1.1
        lab = _labels(g, n + nt, c, zipf)
        x = torch.empty(p, n + nt, device="cuda", dtype=torch.float32)
        x.copy_(proto.T[:, lab])
        for r in range(0, p, 64):
            q = min(p, r + 64)
            x[r:q].add_(torch.randn(q - r, n + nt, generator=g, device="cuda"), alpha=0.3)
        x /= x.norm(dim=0, keepdim=True)
        s["x"], s["xt"] = x.T[:n], x.T[n:]
        s["lab"] = lab[:n]
        # a label vector has every class: the first rows of the training part
        s["lab"][:c] = torch.arange(c, device="cuda")
        s["x"][:c] = proto
    elif kind == "opls":
        n, nt, p, q = case["n"], case["n_test"], case["p"], case["q"]
        x = _lowrank_x(g, n + nt, p, 40, 20.0 * math.sqrt(p), 1.0)
        b1 = _randn(g, p, 40)
        b2 = _randn(g, 40, q) / math.sqrt(p * 40.0)
        y = (x @ b1) @ b2 + 0.1 * _randn(g, n + nt, q)
        s["x"], s["y"], s["xt"] = _colmajor(x[:n]), _colmajor(y[:n]), _colmajor(x[n:])
        s["proj"] = (_randn(g, q, case["dim"]) / math.sqrt(case["dim"])).cpu().numpy()
    else:   # topk
        n, p, c, k = case["n"], case["p"], case["classes"], case["k"]
        k = min(k, p)
        s["xt"] = _randn(g, n, p)
        s["r"] = torch.linalg.qr(_randn(g, p, k))[0].cpu().numpy()
        s["w"] = (_randn(g, k, c) / math.sqrt(k)).cpu().numpy()
        s["mx"] = (0.1 * _randn(g, 1, p)).cpu().numpy()
        s["my"] = (torch.ones(1, c, device="cuda", dtype=torch.float64) / c).cpu().numpy()
        s["bias"] = (0.01 * _randn(g, 1, c)).cpu().numpy().ravel()
    return s


def _slices(case):
    """The component counts of a fit: the largest and fractions of it."""
    k = case["k"]
    want = {1: [k], 2: [max(1, k // 5), k], 3: [max(1, k // 4), max(1, k // 2), k]}[case.get("slices", 1)]
    return sorted(set(want))


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    if kind == "plslda":
        s["codes"] = (s.pop("lab").cpu().numpy() + 1).astype(np.int32)
    elif kind == "dcv":
        s["x"] = _Registered(s["x"])
    elif kind == "cknn":
        s["x"], s["xt"] = _Registered(s["x"]), _Registered(s["xt"])
        s["codes"] = (s.pop("lab").cpu().numpy() + 1).astype(np.int32)
    elif kind == "opls":
        s["xf"] = torch.empty_like(s["x"])        # filtered matrices stay on the device
        s["xtf"] = torch.empty_like(s["xt"])
        s["yp"] = torch.empty(case["q"], case["n_test"], device="cuda", dtype=torch.float64).T
    elif kind == "topk":
        k, c = s["r"].shape[1], case["classes"]
        s["model"] = dict(R=s["r"], W_latent=np.asfortranarray(s["w"][:, :, None]), mX=s["mx"],
                          vX=np.ones_like(s["mx"]), mY=s["my"], m=c, p=case["p"], ncomp=np.array([k]),
                          pls_method="plssvd")
    torch.cuda.synchronize()   # the library works on streams of its own
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "simpls":
        model = lib.pls_model2_fast(s["x"], s["y"], [max(1, case["k"] // 2), case["k"]], seed=1)
        pred = lib.predict_lowrank(model, s["xt"])
        return dict(R=model["R"], Q=model["Q"], mX=model["mX"], mY=model["mY"], B=model["B"], Ypred=pred["Ypred"])
    if kind == "plslda":
        lib.set_precision(case["precision"])
        try:
            r = lib.pls_lda(s["x"], s["y"], s["codes"], s["xt"], _slices(case), case["classes"], method=1,
                            oversample=10, power_iters=2, seed=1)
        finally:
            lib.set_precision("fp64")
        return {k: r[k] for k in ("R", "Q", "mX", "mY", "B", "lda_means", "lda_linear", "lda_constants",
                                  "lda_priors", "lda_lambda", "R_offset", "pred_codes")}
    if kind == "dcv":
        r = lib.double_cv_resident(s["x"].handle, case["n"], s["y"], s["outer"], s["inner"],
                                   np.arange(1, case["k"] + 1), case["classes"], seed=1,
                                   precision=case["precision"])
        return {k: r[k] for k in ("best_comp", "inner_accuracy", "pred", "fit_status")}
    if kind == "cknn":
        return lib.label_aware_cknn_resident(s["x"].handle, s["codes"], case["classes"], s["xt"].handle,
                                             case["n_test"], case["k"], svd_method=4, oversample=10,
                                             power_iters=1, seed=1, knn_k=10, tau=0.2, alpha=0.75, top_m=20,
                                             top_k=5)
    if kind == "opls":
        lib.set_precision(case["precision"])
        try:
            f = lib.opls_filter(s["x"], s["y"], case["north"], out=s["xf"])
            enc = lib.gaussian_y_encode(s["y"], s["proj"])
            model = lib.pls_model2_fast(s["xf"], enc["Z"], [case["k"]], seed=1)
            lib.opls_apply_filter(s["xt"], f["mX"], f["vX"], f["W_orth"], f["P_orth"], out=s["xtf"])
            z = lib.predict_lowrank(model, s["xtf"])["Ypred"][:, :, 0]
            lib.gaussian_y_decode(z, enc["decoder"], enc["y_center"], out=s["yp"])
        finally:
            lib.set_precision("fp64")
        return dict(X=s["xf"], W_orth=f["W_orth"], P_orth=f["P_orth"], Z=enc["Z"], decoder=enc["decoder"],
                    R=model["R"], Q=model["Q"], Ypred=s["yp"])
    return lib.predict_classes(s["model"], s["xt"], class_bias=s["bias"], top_k=min(case["top"], case["classes"]),
                               return_scores=True)


def work(case):
    kind = case["kind"]
    if kind == "simpls":
        n, p, m, k, nt = (case[i] for i in ("n", "p", "m", "k", "n_test"))
        return dict(bytes=8.0 * (n * p + n * m + nt * p + p * k + m * k + 2 * p * m + 2 * nt * m),
                    flops=2.0 * n * p * m + k * (4.0 * n * p + 14.0 * p * m) + 2.0 * nt * p * k)
    if kind == "plslda":
        n, p, c, k, nt = (case[i] for i in ("n", "p", "classes", "k", "n_test"))
        e, sl = (4.0 if case["dtype"] == "float32" else 8.0), len(_slices(case))
        return dict(bytes=e * p * (n + nt) + 8.0 * (n * c + p * k + sl * (p * c + 2 * c * k)) + 4.0 * nt * sl,
                    flops=2.0 * n * p * k + n * p + 10.0 * p * c * (k + 10) + 2.0 * n * k * k + 2.0 * nt * k * (p + c))
    if kind == "dcv":
        n, p, k, c = (case[i] for i in ("n", "p", "k", "classes"))
        fits = case["outer"] * (case["inner"] + 1)
        mult = {"fp64": 1.0, "bf16x3": 3.0, "int8": 15.0}[case["precision"]]
        per = min(2.0 * n * n, 4.0 * n * p) * k * fits      # K products, or two passes over X a component
        gram = mult * n * n * p if 2 * n <= p else 0.0
        return dict(bytes=4.0 * n * p + 8.0 * n * n * (2 * n <= p) + 4.0 * n * (case["outer"] + 3),
                    flops=gram + per + fits * k * n * 6.0 * c)
    if kind == "cknn":
        n, p, k, c, nt = (case[i] for i in ("n", "p", "k", "classes", "n_test"))
        # 20 candidate classes a test row, each of the mean class size
        return dict(bytes=4.0 * p * (n + nt) + 4.0 * n + nt * 5 * 12.0,
                    flops=2.0 * n * p * k + n * p + 2.0 * n * k * k + 2.0 * nt * k * c + nt * 20 * (n / c) * 2.0 * k)
    if kind == "opls":
        n, p, q, d, k, nt = (case[i] for i in ("n", "p", "q", "dim", "k", "n_test"))
        return dict(bytes=8.0 * (2 * n * p + n * q + 2 * nt * p + nt * q + n * d + q * d + p * k),
                    flops=2.0 * n * p * (case["north"] * (q + 6) + d + 2 * k) + 4.0 * n * q * d + 2.0 * nt * d * q)
    n, p, k, c = (case[i] for i in ("n", "p", "k", "classes"))
    return dict(bytes=8.0 * (n * p + p * k + k * c) + 12.0 * n * case["top"], flops=2.0 * n * k * (p + c))


# ---------------------------------------------------- the same in 64 bits ---
def _sketch(count, seed):
    """`count` standard normal values as the seeded sketches draw them: 32-bit
    Mersenne Twister, two draws a uniform, Marsaglia's polar method (the second
    coordinate first)."""
    bits = np.random.MT19937()
    bits._legacy_seeding(int(seed) & 0xFFFFFFFF)
    got, have = [], 0
    while have < count:
        trials = int((count - have) * 0.7) + 64
        raw = bits.random_raw(4 * trials).astype(np.float64).reshape(trials, 2, 2)
        u = (raw[:, :, 0] + raw[:, :, 1] * 4294967296.0) / 18446744073709551616.0
        xy = 2.0 * u - 1.0
        r2 = xy[:, 0] ** 2 + xy[:, 1] ** 2
        ok = (r2 <= 1.0) & (r2 != 0.0)
        mult = np.sqrt(-2.0 * np.log(r2[ok]) / r2[ok])
        z = np.stack([xy[ok, 1] * mult, xy[ok, 0] * mult], axis=1).ravel()
        got.append(z)
        have += z.size
    return torch.from_numpy(np.concatenate(got)[:count]).cuda()


def _simpls64(x, y, k, seed):
    """Fast SIMPLS on centred x, y: one vector a component, refreshed by two
    power iterations from the last one (the first from the seeded sketch)."""
    p, m = x.shape[1], y.shape[1]
    s = x.T @ y
    rr, qq, vv = x.new_zeros(p, k), x.new_zeros(m, k), x.new_zeros(p, k)
    w = _sketch(p, seed) if m > 1 else s[:, 0].clone()
    for a in range(k):
        if m == 1:
            w = s[:, 0].clone()
        else:
            for _ in range(2):
                w = s @ (s.T @ w)
        r = w / w.norm()
        r = torch.where(r[0] >= 0, -r, r)
        t = x @ r
        tn = t.norm()
        t, r = t / tn, r / tn
        load = x.T @ t
        v = load - vv[:, :a] @ (vv[:, :a].T @ load)
        v = v / v.norm()
        s = s - torch.outer(v, v @ s)
        rr[:, a], qq[:, a], vv[:, a] = r, y.T @ t, v
        w = r
    return rr, qq


def _rsvd64(s, k, power, seed):
    """The seeded randomized SVD (oversampling 10), or the exact one where the
    sketch would not be smaller than the matrix."""
    small = min(s.shape)
    if small < 6 or k + 10 >= small:
        u, d, vh = torch.linalg.svd(s, full_matrices=False)
        return u[:, :k], d[:k], vh[:k].T
    y = s @ _sketch(s.shape[1] * (k + 10), seed).reshape(k + 10, s.shape[1]).T
    if power == 1:
        y = s @ (s.T @ y)
    else:
        for _ in range(power):
            y = s @ torch.linalg.qr(s.T @ y)[0]
    q = torch.linalg.qr(y)[0]
    b = q.T @ s
    u, d, vh = torch.linalg.svd(b, full_matrices=False)
    return q @ u[:, :k], d[:k], vh[:k].T


def _exact_simpls(case, s):
    x, y, k = s["x"], s["y"], case["k"]
    mx, my = x.mean(dim=0), y.mean(dim=0)
    r, q = _simpls64(x - mx, y - my, k, 1)
    nc = [max(1, k // 2), k]
    t = (s["xt"] - mx) @ r
    return dict(R=r, Q=q, mX=mx[None, :], mY=my[None, :], B=torch.stack([r[:, :c] @ q[:, :c].T for c in nc], dim=2),
                Ypred=torch.stack([t[:, :c] @ q[:, :c].T + my for c in nc], dim=2))


def _exact_plslda(case, s):
    # latent vectors are defined up to their sign: only what does not depend on
    # the signs has a value of its own
    x, y, lab, c = s["x"].double(), s["y"], s["lab"], case["classes"]
    n, p = x.shape
    mx, my = x.mean(dim=0), y.mean(dim=0)
    xc, yc = x - mx, y - my
    sxy = xc.T @ yc
    if min(n, p, c) <= 32:
        u, d, vh = torch.linalg.svd(sxy, full_matrices=False)
        u, d, v = u[:, :case["k"]], d[:case["k"]], vh[:case["k"]].T
    else:
        u, d, v = _rsvd64(sxy, case["k"], 2, 1)
    t = xc @ u
    gram = t.T @ t
    count = torch.bincount(lab, minlength=c).double()
    mean = x.new_zeros(c, t.shape[1]).index_add_(0, lab, t) / count[:, None]
    pooled = (gram - (mean * count[:, None]).T @ mean) / max(1.0, float(n - c))
    nc = _slices(case)
    tt = (s["xt"].double() - mx) @ u
    bs, const, lam, pred = [], [], [], []
    for k in nc:
        bs.append(u[:, :k] @ torch.linalg.solve(gram[:k, :k], torch.diag(d[:k])) @ v[:, :k].T)
        pk = pooled[:k, :k]
        ridge = 1e-8 * torch.trace(pk) / k
        lin = torch.linalg.solve(pk + ridge * torch.eye(k, device="cuda", dtype=torch.float64), mean[:, :k].T).T
        const.append(-0.5 * (mean[:, :k] * lin).sum(dim=1) + torch.log(count / n))
        lam.append(ridge)
        pred.append((tt[:, :k] @ lin.T + const[-1]).argmax(dim=1).int() + 1)
    return dict(R=None, Q=None, mX=mx[None, :], mY=my[None, :], B=torch.stack(bs, dim=2), lda_means=None,
                lda_linear=None, lda_constants=torch.stack(const, dim=1), lda_priors=count / n,
                lda_lambda=torch.stack(lam), R_offset=None, pred_codes=torch.stack(pred, dim=1))


def _exact_dcv(case, s):
    x, y = s["x"].double(), torch.from_numpy(s["y"]).cuda().long() - 1
    n, c, k = case["n"], case["classes"], case["k"]
    outer, inner = torch.from_numpy(s["outer"]).cuda(), torch.from_numpy(np.array(s["inner"])).cuda()
    ko = int(outer.max()) + 1
    hot = torch.nn.functional.one_hot(y, c).double()

    def labels(train, test, comps, seed):
        """Predicted classes of the test rows at each component count."""
        xa, ya = x[train], hot[train]
        mx, my = xa.mean(dim=0), ya.mean(dim=0)
        r, q = _simpls64(xa - mx, ya - my, comps, seed)
        t = (x[test] - mx) @ r
        scores = torch.cumsum(t[:, None, :] * q[None, :, :], dim=2) + my[None, :, None]
        return scores.argmax(dim=1)

    best = np.zeros(ko, dtype=np.int32)
    acc = np.zeros((ko, k))
    pred = torch.zeros(n, dtype=torch.int32, device="cuda")
    for o in range(ko):
        rows = torch.nonzero(outer != o)[:, 0]
        test = torch.nonzero(outer == o)[:, 0]
        hits = torch.zeros(k, dtype=torch.float64, device="cuda")
        for f in range(int(inner[rows, o].max()) + 1):
            out = rows[inner[rows, o] == f]
            lab = labels(rows[inner[rows, o] != f], out, k, 1 + 1000 + o + 1 + f)
            hits += (lab == y[out][:, None]).double().sum(dim=0)
        a = (hits / rows.numel()).cpu().numpy()
        acc[o], best[o] = a, int(np.argmax(a)) + 1
        pred[test] = labels(rows, test, int(best[o]), 1 + 2000 + o + 1)[:, -1].int() + 1
    return dict(best_comp=best, inner_accuracy=acc, pred=pred, fit_status=None)


def _exact_cknn(case, s):
    n, p, c, k, nt = (case[i] for i in ("n", "p", "classes", "k", "n_test"))
    lab = s["lab"]
    step = 100_000
    blocks = [(i, min(n, i + step)) for i in range(0, n, step)]
    mx = sum(s["x"][a:b].double().sum(dim=0) for a, b in blocks) / n
    sums = torch.zeros(c, p, device="cuda", dtype=torch.float64)
    for a, b in blocks:
        sums.index_add_(0, lab[a:b], s["x"][a:b].double() - mx)
    share = torch.bincount(lab, minlength=c).double() / n
    sxy = sums.T - torch.outer(sums.sum(dim=0), share)
    u, d, _ = _rsvd64(sxy, k, 1, 1)
    t = torch.cat([(s["x"][a:b].double() - mx) @ u for a, b in blocks])
    gram = t.T @ t
    ridge = 1e-10 * gram.diagonal().mean()
    coef = torch.linalg.solve(gram + ridge * torch.eye(k, device="cuda", dtype=torch.float64), torch.diag(d))
    unit = lambda m: m / m.norm(dim=1, keepdim=True)  # noqa: E731
    t = unit(t @ coef)
    new = unit(((s["xt"].double() - mx) @ u) @ coef)
    count = torch.bincount(lab, minlength=c).clamp(min=1).double()
    cent = unit(torch.zeros(c, k, device="cuda", dtype=torch.float64).index_add_(0, lab, t) / count[:, None])
    base, cand = (new @ cent.T).topk(20, dim=1)
    score = torch.full_like(base, -math.inf)
    order = torch.argsort(lab)
    ends = torch.cumsum(torch.bincount(lab, minlength=c), 0).tolist()
    for cls in range(c):
        i, j = torch.nonzero(cand == cls, as_tuple=True)
        members = t[order[(ends[cls - 1] if cls else 0):ends[cls]]]
        rows = max(1, 400_000_000 // max(1, members.shape[0]))
        for a in range(0, i.numel(), rows):
            sim = new[i[a:a + rows]] @ members.T
            near = sim.topk(min(10, members.shape[0]), dim=1).values
            smooth = near[:, 0] + 0.2 * torch.log(torch.exp((near - near[:, :1]) / 0.2).mean(dim=1))
            score[i[a:a + rows], j[a:a + rows]] = smooth + 0.75 * base[i[a:a + rows], j[a:a + rows]]
    val, at = score.topk(5, dim=1)
    return dict(top_index=(torch.gather(cand, 1, at) + 1).int(), top_score=val)


def _exact_opls(case, s):
    x, y, xt = s["x"], s["y"], s["xt"]
    mx, my = x.mean(dim=0), y.mean(dim=0)
    xf, yc, xtf = x - mx, y - my, xt - mx
    for _ in range(case["north"]):
        sxy = xf.T @ yc
        w = sxy @ torch.linalg.eigh(sxy.T @ sxy).eigenvectors[:, -1]
        w = w / w.norm()
        t = xf @ w
        load = xf.T @ t / (t @ t)
        wo = load - w * (w @ load)
        wo = wo / wo.norm()
        to = xf @ wo
        po = xf.T @ to / (to @ to)
        xf = xf - torch.outer(to, po)
        xtf = xtf - torch.outer(xtf @ wo, po)
    g = torch.from_numpy(s["proj"]).cuda()
    z = yc @ g
    ztz = z.T @ z
    ridge = 1e-8 * ztz.diagonal().mean()
    dec = torch.linalg.solve(ztz + ridge * torch.eye(ztz.shape[0], device="cuda", dtype=torch.float64), z.T @ yc)
    m2, mz = xf.mean(dim=0), z.mean(dim=0)
    r, q = _simpls64(xf - m2, z - mz, case["k"], 1)
    zp = ((xtf - m2) @ r) @ q.T + mz
    # the filter's directions are defined up to their sign; the trailing SIMPLS
    # directions lie in the noise and follow the rounding of the products
    return dict(X=xf, W_orth=None, P_orth=None, Z=z, decoder=dec, R=None, Q=None, Ypred=zp @ dec + my)


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "topk":
        cu = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
        sc = ((s["xt"] - cu(s["mx"])) @ cu(s["r"])) @ cu(s["w"]) + cu(s["my"]) + cu(s["bias"])
        val, at = sc.topk(min(case["top"], case["classes"]), dim=1)
        return dict(top_index=(at + 1).int()[:, :, None], top_score=val[:, :, None])
    return {"simpls": _exact_simpls, "plslda": _exact_plslda, "dcv": _exact_dcv, "cknn": _exact_cknn,
            "opls": _exact_opls}[kind](case, s)
