"""The work that users of this package have it do, as cases that can be timed.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)`
one more of the same ranges, `prepare(case, seed)` what a program holds before
the call, `run(state)` one call through the package's public entry points,
`work(case)` the bytes and operations the call cannot do without, and
`exact(case, seed)` the same outputs computed in 64 bits with numpy, where the
outputs are a closed formula of the inputs (a Levenberg-Marquardt fit of tens
of iterations is not: it amplifies any rounding).

Objects are seeded synthetic asteroids (`ps_claude_opt_b200.synth`): convex
bodies seen as relative lightcurves and, in some, calibrated sparse points.
"""
from __future__ import annotations

import math

import numpy as np

N_POLES = 10
STEP_SEEDS = 7919  # spacing of the seeds of one case's objects

# Sizes of the objects: the package's configuration 1, its production object
# (with and without the calibrated points) and its largest models.
CONFIG1 = dict(l_max=3, m_max=3, nrows=6, curves=20, pts_lo=60, pts_hi=60, sparse=0, sparse_curves=1, stop=50.0)
PRODUCTION = dict(l_max=6, m_max=6, nrows=8, curves=40, pts_lo=50, pts_hi=120, sparse=400, sparse_curves=2, stop=50.0)
RELATIVE = dict(PRODUCTION, sparse=0)
LARGEST = dict(l_max=8, m_max=8, nrows=10, curves=110, pts_lo=90, pts_hi=90, sparse=0, sparse_curves=1, stop=0.005)


def listed():
    return [
        # One evaluation of the model: chi^2, its gradient and J^T W J at given
        # parameters.  What a host that drives its own optimiser, maps chi^2
        # over a pole grid or checks a solution calls, thousands of times.
        dict(name="eval-config1", kind="eval", **CONFIG1),
        dict(name="eval-production", kind="eval", **PRODUCTION),
        # All poles of one trial frequency, 50 iterations each: the smallest
        # fit call, e.g. a line refitted by hand.
        dict(name="fit-one-frequency", kind="fit", precision="fp64", freqs=1, **PRODUCTION),
        # The FP64 refits that end a mixed-precision screened scan: the handle
        # is configured again for FP64, then about 30 frequencies are fitted.
        dict(name="refit-candidates", kind="refit", precision="fp64", freqs=31, **PRODUCTION),
        # A stretch of the full scan of the production object, as the host
        # program makes it between two checkpoints.
        dict(name="scan-production", kind="scan", freqs=61, **PRODUCTION),
        # The largest models, fits that run until the rms stops improving.
        dict(name="scan-largest", kind="scan", freqs=37, **LARGEST),
        # The mixed-precision first pass of a screened scan.
        dict(name="fit-mixed", kind="fit", precision="mixed", freqs=59, **RELATIVE),
        # A whole small object: convexity-weight search, then the scan.
        dict(name="search-config1", kind="search", freqs=60, **CONFIG1),
        # Several objects of different sizes in one call.
        dict(name="batch-mixed-sizes", kind="batch", first=0, objects=6, freqs=3),
        # The screen: features of every trial frequency of the production grid ...
        dict(name="screen-features", kind="features", freqs=5000, **PRODUCTION),
        # ... the network's scores of them ...
        dict(name="screen-scores", kind="predict", rows=5000),
        # ... and one step of its training.
        dict(name="screen-train-step", kind="train", rows=1024),
    ]


# ------------------------------------------------------------------ draws

KINDS = ("eval", "fit", "fit", "refit", "scan", "scan", "mixed", "search", "batch", "noalloc", "features", "predict",
         "train")


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_object(rng, l_top=8):
    l_max = rng.randint(3, l_top)
    m_max = l_max if rng.random() < 0.7 else rng.randint(2, l_max)
    nrows = rng.randint(5, 10)
    points = _log_uniform(rng, 300, 12000)
    curves = max(4, min(150, int(points / rng.uniform(30, 110))))
    mean = points / curves
    lo = max(3, int(mean * rng.uniform(0.5, 1.0)))
    hi = max(lo, int(2 * mean - lo))
    sparse = 0 if rng.random() < 0.5 else rng.randint(20, 500)
    stop = rng.choice([50.0, 50.0, 20.0, 0.005, 0.02])
    return dict(l_max=l_max, m_max=m_max, nrows=nrows, curves=curves, pts_lo=lo, pts_hi=hi, sparse=sparse,
                sparse_curves=1 + (sparse > 200), stop=stop)


def draw(rng):
    top = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(KINDS)
        if kind == "eval":
            case = dict(kind="eval", **_draw_object(rng))
        elif kind in ("fit", "refit"):
            case = dict(kind=kind, precision="fp64", freqs=int(round(_log_uniform(rng, 1, 150))), **_draw_object(rng))
        elif kind == "mixed":
            case = dict(kind=rng.choice(["fit", "refit"]), precision="mixed", freqs=int(round(_log_uniform(rng, 1, 150))),
                        **_draw_object(rng, 6))
        elif kind in ("scan", "search"):
            case = dict(kind=kind, freqs=int(round(_log_uniform(rng, 5, 300))), **_draw_object(rng))
        elif kind == "noalloc":
            case = dict(kind="noalloc", freqs=int(round(_log_uniform(rng, 1, 20))), **_draw_object(rng, 6))
        elif kind == "batch":
            case = dict(kind="batch", first=rng.randrange(60), objects=rng.randint(2, 6), freqs=rng.randint(1, 6))
        elif kind == "features":
            case = dict(kind="features", freqs=int(round(_log_uniform(rng, 200, 12000))), **_draw_object(rng))
        else:
            case = dict(kind=kind, rows=int(round(_log_uniform(rng, 64, 12000 if kind == "predict" else 4096))))
        if work(case)["flops"] <= 0.9 * top:
            return case


# ------------------------------------------------------------------ inputs


def _config(case):
    from ps_claude_opt_b200 import synth

    # the truth brightness on 30 x 60 directions: finer than any fit's facets,
    # and short to generate
    return synth.SynthConfig(l_max=case["l_max"], m_max=case["m_max"], nrows=case["nrows"], n_dense=case["curves"],
                             dense_pts=(case["pts_lo"], case["pts_hi"]), n_sparse=case["sparse"],
                             sparse_curves=case["sparse_curves"], n_freq=max(400, case.get("freqs", 1)),
                             stop_condition=case["stop"], truth_grid=(30, 60))


def _object(case, seed):
    from ps_claude_opt_b200 import objects, synth

    return objects.parse_input(synth.generate(_config(case), seed)[0])


def _batch_configs(case):
    from ps_claude_opt_b200 import synth

    return [synth.config3_object(case["first"] + k)[0] for k in range(case["objects"])]


def _parameters(obj, seed):
    """A parameter vector as met inside a fit: the start values of one trial
    frequency and pole, moved."""
    from ps_claude_opt_b200 import objects

    rng = np.random.default_rng(seed + 1)
    a = objects.initial_params(obj, int(rng.integers(1, obj.grid.n_max + 1)), int(rng.integers(0, N_POLES)))
    nc = obj.n_coef
    top = np.abs(obj.dsph.reshape(obj.n_fac, nc)).max(axis=0)  # the basis is not normalised
    a[2:nc + 1] += rng.normal(0.0, 0.05, nc - 1) / np.maximum(top[1:], 1e-3)
    a[nc + 1:nc + 3] += rng.normal(0.0, 0.1, 2)
    a[nc + 4:nc + 7] *= 1.0 + rng.normal(0.0, 0.05, 3)
    a[nc + 7] += rng.normal(0.0, 0.1)
    return a


def _items(case, obj, seed):
    """All poles of `freqs` consecutive trial frequencies of the grid."""
    n = case["freqs"]
    first = 1 + int(np.random.default_rng(seed + 2).integers(0, obj.grid.n_max - n + 1))
    return (np.repeat(np.arange(first, first + n), N_POLES).astype(np.int32),
            np.tile(np.arange(N_POLES), n).astype(np.int32))


def _network_arrays(seed, rows):
    """Features as the screen's normalisation leaves them, and targets."""
    rng = np.random.default_rng(seed + 3)
    return rng.standard_normal((rows, 88)).astype(np.float32), rng.standard_normal(rows).astype(np.float32)


def _network(seed):
    """The screening network in the middle of its training."""
    import torch

    from ps_claude_opt_b200 import screen

    net = screen.Mlp(seed=seed)
    rng = np.random.default_rng(seed + 4)
    for w, m, v in zip(net.W + net.b, net.mW + net.mb, net.vW + net.vb):
        shape = tuple(w.shape)
        m.copy_(torch.from_numpy(rng.normal(0.0, 1e-3, shape).astype(np.float32)))
        v.copy_(torch.from_numpy(rng.uniform(1e-6, 1e-5, shape).astype(np.float32)))
    for b in net.b:
        b.copy_(torch.from_numpy(rng.normal(0.0, 0.05, tuple(b.shape)).astype(np.float32)))
    net.steps = 200
    return net


def prepare(case, seed):
    kind = case["kind"]
    if kind == "predict":
        return dict(kind=kind, net=_network(seed), x=_network_arrays(seed, case["rows"])[0])
    if kind == "train":
        import torch

        x, y = _network_arrays(seed, case["rows"])
        return dict(kind=kind, net=_network(seed), x=torch.from_numpy(x).cuda().to(torch.bfloat16),
                    y=torch.from_numpy(y).cuda())
    if kind == "batch":
        from ps_claude_opt_b200 import objects, synth

        objs = [objects.parse_input(synth.generate(c, seed + STEP_SEEDS * k)[0])
                for k, c in enumerate(_batch_configs(case))]
        return dict(kind=kind, objs=objs, freqs=case["freqs"])
    obj = _object(case, seed)
    if kind == "features":
        from ps_claude_opt_b200 import screen

        return dict(kind=kind, obj=obj, freqs=screen.frequencies(obj, 1, case["freqs"]))
    if kind == "search":
        return dict(kind=kind, obj=obj, freqs=case["freqs"])
    if kind == "noalloc":
        return dict(kind=kind, obj=obj, items=_items(case, obj, seed))
    from ps_claude_opt_b200 import native

    eng = native.Engine(obj)
    if case.get("precision") == "mixed":
        eng.set_precision(native.PRECISION_MIXED)
    state = dict(kind=kind, obj=obj, eng=eng)
    if kind == "eval":
        eng.configure()
        state["a"] = _parameters(obj, seed)
    elif kind == "fit":
        eng.configure()
        state["items"] = _items(case, obj, seed)
    elif kind == "refit":
        state["items"] = _items(case, obj, seed)
    elif kind == "scan":
        state["first"] = int(_items(case, obj, seed)[0][0])
        state["freqs"] = case["freqs"]
    return state


def run(state):
    from ps_claude_opt_b200 import native, screen

    kind = state["kind"]
    if kind == "eval":
        chisq, alpha, beta, area = state["eng"].eval(state["a"])
        return dict(chisq=chisq, alpha=alpha, beta=beta, area=area)
    if kind == "fit":
        return state["eng"].fit_items(*state["items"])
    if kind == "refit":
        state["eng"].configure()
        return state["eng"].fit_items(*state["items"])
    if kind == "scan":
        return state["eng"].start(state["obj"].conw_r, n_start_from=state["first"], max_lines=state["freqs"])
    if kind == "search":
        return native.run_object(state["obj"], max_freq=state["freqs"])
    if kind == "noalloc":
        return native.fit_items_noalloc(state["obj"], *state["items"])
    if kind == "batch":
        return native.scan_batch(state["objs"], max_freq=state["freqs"])
    if kind == "features":
        return screen.features(state["obj"], state["freqs"])
    if kind == "predict":
        return state["net"].predict(state["x"])
    net = state["net"]
    loss = net.train_step(state["x"], state["y"], 1e-3)
    return dict(loss=loss, W=net.W, b=net.b)


# ------------------------------------------------------------------ work


def _n_coef(l_max, m_max):
    return sum((2 if m else 1) for m in range(m_max + 1) for _ in range(m, l_max + 1))


def _fit_sizes(l_max, m_max, nrows, points, n_curves, rel_only):
    nc = _n_coef(l_max, m_max)
    mfit = nc + 7 - (1 if rel_only else 0)
    nf = 8 * nrows * nrows
    tables = 8.0 * (points * 9 + nf * (nc + 4) + n_curves * 3 + nc)
    return nc, mfit, nf, tables


def _fit_flops(nc, mfit, nf, points, iterations):
    """A point sees about 0.45 of the facets.  Every trial step needs chi^2,
    i.e. the brightness; the derivatives are needed where the step is taken
    (a little under half of the steps, and the start)."""
    seen = 0.45 * nf
    bright = points * (150 + 10 * nf + 30 * seen) + nf * (2 * nc + 2)
    deriv = points * (seen * (30 + 2 * nc) + mfit * (mfit + 1) + 8 * mfit) + 6 * nf * nc
    return (iterations + 1) * bright + (1 + 0.45 * iterations) * deriv + iterations * 2.0 / 3 * mfit ** 3


def _iterations(stop):
    return int(stop) if stop > 1 else 11  # converging fits take 10 (the minimum) to 13


def work(case):
    kind = case["kind"]
    layers = (88, 256, 256, 256, 1)
    macs = sum(k * n for k, n in zip(layers[:-1], layers[1:]))
    weights = macs + sum(layers[1:])
    if kind == "predict":
        return dict(bytes=4.0 * (88 + 1) * case["rows"] + 2.0 * weights, flops=2.0 * macs * case["rows"])
    if kind == "train":
        # forward, and the two products of the backward pass (one for the first layer)
        return dict(bytes=2.0 * 88 * case["rows"] + 4.0 * case["rows"] + (4 * 6 + 4) * weights,
                    flops=2.0 * (3 * macs - layers[0] * layers[1]) * case["rows"])
    if kind == "batch":
        b = f = 0.0
        for c in _batch_configs(case):
            points = c.n_dense * c.dense_pts[0]
            nc, mfit, nf, tables = _fit_sizes(c.l_max, c.m_max, c.nrows, points, c.n_dense, True)
            # two rounds of the convexity-weight search (100 fits each), then the scan
            f += (200 + N_POLES * case["freqs"]) * _fit_flops(nc, mfit, nf, points, _iterations(c.stop_condition))
            b += tables
        return dict(bytes=b, flops=f)
    points = case["curves"] * (case["pts_lo"] + case["pts_hi"]) / 2 + case["sparse"]
    n_curves = case["curves"] + (case["sparse_curves"] if case["sparse"] else 0)
    if kind == "features":
        # four folds of every point (its own curve's; all; first or second half),
        # the statistics of 64 bins of every curve and fold
        return dict(bytes=12.0 * points + case["freqs"] * (8.0 + 4 * 88),
                    flops=case["freqs"] * (points * 3 * 8.0 + (n_curves + 3) * (64 * 4 * 6.0 + 32 * 16)))
    nc, mfit, nf, tables = _fit_sizes(case["l_max"], case["m_max"], case["nrows"], points, n_curves,
                                      case["sparse"] == 0)
    if kind == "eval":
        return dict(bytes=tables + 8.0 * mfit * (mfit + 1), flops=_fit_flops(nc, mfit, nf, points, 0))
    fits = N_POLES * case["freqs"] + (200 if kind == "search" else 0)
    return dict(bytes=tables + 64.0 * fits, flops=fits * _fit_flops(nc, mfit, nf, points, _iterations(case["stop"])))


# ------------------------------------------------------------------ exact values


def _exact_eval(obj, a):
    """chi^2, J^T W J, J^T W dy and the summed facet area at the 1-based
    parameter vector a: the convex-body brightness model in 64 bits."""
    nc, ma, nf, n_pts = obj.n_coef, obj.ma, obj.n_fac, obj.n_points
    normal = obj.normal.reshape(nf, 3)
    basis = obj.dsph.reshape(nf, nc)
    area = obj.d_area * np.exp(basis @ a[1:nc + 1])
    bet, lam, om, pa, pd, pk = a[nc + 1:nc + 7]
    cl, cls = math.exp(a[ma - 1]), a[ma]
    sb, cb, sl, cl_ = math.sin(bet), math.cos(bet), math.sin(lam), math.cos(lam)
    rot = np.array([[cb * cl_, cb * sl, -sb], [-sl, cl_, 0], [sb * cl_, sb * sl, cb]])
    rot_b = np.array([[-sb * cl_, -sb * sl, -cb], [0, 0, 0], [cb * cl_, cb * sl, -sb]])
    rot_l = np.array([[-cb * sl, cb * cl_, 0], [-cl_, -sl, 0], [-sb * sl, sb * cl_, 0]])
    rows = np.zeros((n_pts, ma + 1))
    for p0 in range(0, n_pts, 2048):
        sl_ = slice(p0, min(n_pts, p0 + 2048))
        t = obj.tim[sl_]
        f = om * t + obj.phi0
        f = f - 2 * math.pi * np.round(f / (2 * math.pi))
        c, s = np.cos(f), np.sin(f)

        def spin(v, cc, ss, z):
            return np.stack([cc * v[:, 0] + ss * v[:, 1], -ss * v[:, 0] + cc * v[:, 1], z * v[:, 2]], axis=1)

        both = [obj.ee.reshape(n_pts, 3)[sl_], obj.ee0.reshape(n_pts, 3)[sl_]]
        e, e0 = (spin(v @ rot.T, c, s, 1.0) for v in both)
        d_pole = [[spin(v @ m.T, c, s, 1.0) for v in both] for m in (rot_b, rot_l)]
        d_spin = [spin(v @ rot.T, -s * t, c * t, 0.0) for v in both]
        alpha = np.arccos(np.clip(np.sum(both[0] * both[1], axis=1), -1, 1))
        ff = np.exp(-alpha / pd)
        scale = 1 + pa * ff + pk * alpha
        mu, mu0 = e @ normal.T, e0 @ normal.T
        vis = (mu > 1e-8) & (mu0 > 1e-8)
        mu, mu0 = np.where(vis, mu, 0.0), np.where(vis, mu0, 0.0)
        den = np.where(vis, mu + mu0, 1.0)
        w = area * (mu * mu0 * (cl + cls / den))
        g = area * (cls * (mu0 / den) ** 2 + cl * mu0) * vis
        g0 = area * (cls * (mu / den) ** 2 + cl * mu) * vis
        u, u0 = g @ normal, g0 @ normal
        br = w.sum(axis=1)
        r = rows[sl_]
        r[:, :nc] = scale[:, None] * (w @ basis)
        for k, (d, d0) in enumerate(d_pole + [d_spin]):
            r[:, nc + k] = scale * (np.sum(d * u, axis=1) + np.sum(d0 * u0, axis=1))
        r[:, nc + 3] = br * ff
        r[:, nc + 4] = br * pa * ff * alpha / (pd * pd)
        r[:, nc + 5] = br * alpha
        r[:, nc + 6] = scale * cl * ((mu * mu0) @ area)
        r[:, nc + 7] = scale * ((mu * mu0 / den) @ area)
        r[:, nc + 8] = scale * br
    dy = np.array(obj.brightness, dtype=np.float64)
    jac = rows[:, :ma].copy()
    q = 0
    for n, rel in zip(obj.curve_len, obj.curve_rel):
        k = slice(q, q + n)
        q += n
        ym = rows[k, ma]
        if rel:
            tot = ym.sum()
            coef = obj.sig[k.start] * n / tot
            jac[k] = coef * (rows[k, :ma] - (ym / tot)[:, None] * rows[k, :ma].sum(axis=0))
            ym = coef * ym
        dy[k] -= ym
    weight = obj.sigr2 * obj.weight
    # the three pseudo-points of the convexity regularisation
    jac = np.vstack([jac, np.zeros((3, ma))])
    jac[n_pts:, :nc] = (area[:, None] * normal).T @ basis
    dy = np.concatenate([dy, -(area @ normal)])
    weight = np.concatenate([weight, np.full(3, obj.conw_r ** 2)])
    jac = jac[:, np.flatnonzero(obj.ia[1:])]
    return dict(chisq=float(np.sum(weight * dy * dy)), alpha=(jac * weight[:, None]).T @ jac,
                beta=jac.T @ (weight * dy), area=float(area.sum()))


def _fold_stats(cnt, s1, s2):
    """The 8 statistics of folds given as [..., 64] bin counts, sums and sums
    of squares: within-bin over total variance for 64, 32, 16 and 8 bins, and
    the shares of four harmonics in the 32-bin mean curve."""
    out = np.zeros(cnt.shape[:-1] + (8,))
    n, a, q = cnt.sum(-1), s1.sum(-1), s2.sum(-1)
    total = q - np.where(n > 0, a * a / np.maximum(n, 1), 0.0)
    for lev in range(4):
        shape = cnt.shape[:-1] + (64 >> lev, 1 << lev)
        c, m, qq = (v.reshape(shape).sum(-1) for v in (cnt, s1, s2))
        within = np.where(c > 0, qq - m * m / np.maximum(c, 1), 0.0).sum(-1)
        out[..., lev] = np.where(total > 0, within / np.where(total > 0, total, 1.0), 1.0)
    shape = cnt.shape[:-1] + (32, 2)
    c, m = cnt.reshape(shape).sum(-1), s1.reshape(shape).sum(-1)
    mean = np.where(c > 0, m / np.maximum(c, 1), 0.0)
    ang = 2 * np.pi * np.outer(np.arange(32), np.arange(1, 5)) / 32
    pw = (mean @ np.cos(ang)) ** 2 + (mean @ np.sin(ang)) ** 2
    tot = pw.sum(-1, keepdims=True)
    out[..., 4:] = np.where(tot > 0, pw / np.where(tot > 0, tot, 1.0), 0.25)
    return out


def _exact_features(obj, freqs):
    n_curves = len(obj.curve_len)
    curve = np.repeat(np.arange(n_curves), obj.curve_len)
    mean = np.bincount(curve, obj.brightness) / obj.curve_len
    y = obj.brightness / mean[curve] - 1.0
    t_mid = 0.5 * (obj.tim.min() + obj.tim.max())
    # folds: every curve, all points, the first half of the time span, the second
    half = np.where(obj.tim < t_mid, n_curves + 1, n_curves + 2)
    folds = n_curves + 3
    fold = np.concatenate([curve, np.full(len(y), n_curves), half]) * 64
    yy = np.tile(y, 3)
    y2 = yy * yy
    out = np.zeros((len(freqs), 88))
    w = np.asarray(obj.curve_len, dtype=np.float64)
    for f0 in range(0, len(freqs), 64):
        fs = freqs[f0:f0 + 64]
        hist = np.zeros((3, len(fs), folds * 64))
        for i, f in enumerate(fs):
            ph = obj.tim * (24.0 * f)
            b = np.clip(((ph - np.floor(ph)) * 64).astype(np.int64), 0, 63)
            at = fold + np.tile(b, 3)
            hist[0, i] = np.bincount(at, minlength=folds * 64)
            hist[1, i] = np.bincount(at, yy, minlength=folds * 64)
            hist[2, i] = np.bincount(at, y2, minlength=folds * 64)
        st = _fold_stats(*hist.reshape(3, len(fs), folds, 64))
        per = st[:, :n_curves]
        srt = np.sort(per, axis=1)
        agg = np.zeros((len(fs), 8, 8))
        agg[..., 0] = np.einsum("fcs,c->fs", per, w) / w.sum()
        agg[..., 1] = per.mean(axis=1)
        agg[..., 2] = per.std(axis=1)
        agg[..., 3] = srt[:, 0]
        for k, qf in ((4, 0.25), (5, 0.5), (6, 0.75)):
            pos = qf * (n_curves - 1)
            lo = int(math.floor(pos))
            hi = min(lo + 1, n_curves - 1)
            agg[..., k] = srt[:, lo] + (pos - lo) * (srt[:, hi] - srt[:, lo])
        agg[..., 7] = srt[:, -1]
        out[f0:f0 + len(fs), :64] = agg.reshape(len(fs), 64)
        out[f0:f0 + len(fs), 64:] = st[:, n_curves:].reshape(len(fs), 24)
    return out


def _forward(W, b, x):
    h = [x]
    for l, (w, c) in enumerate(zip(W, b)):
        z = h[-1] @ w.T + c
        h.append(np.maximum(z, 0.0) if l < len(W) - 1 else z)
    return h


def exact(case, seed):
    kind = case["kind"]
    if kind == "eval":
        obj = _object(case, seed)
        return _exact_eval(obj, _parameters(obj, seed))
    if kind == "features":
        from ps_claude_opt_b200 import screen

        obj = _object(case, seed)
        return _exact_features(obj, screen.frequencies(obj, 1, case["freqs"]))
    if kind not in ("predict", "train"):
        return None
    net = _network(seed)
    W, b, mW, mb, vW, vb = ([np.asarray(t.cpu().numpy(), dtype=np.float64) for t in ts]
                            for ts in (net.W, net.b, net.mW, net.mb, net.vW, net.vb))
    x, y = (v.astype(np.float64) for v in _network_arrays(seed, case["rows"]))
    if kind == "predict":
        return _forward(W, b, x)[-1][:, 0]
    h = _forward(W, b, x)
    diff = h[-1][:, 0] - y
    dz = (2.0 / len(y)) * diff[:, None]
    step = net.steps + 1
    for l in range(len(W) - 1, -1, -1):
        gW, gb = dz.T @ h[l], dz.sum(axis=0)
        if l > 0:
            dz = (dz @ W[l]) * (h[l] > 0)
        for w, g, m, v in ((W[l], gW, mW[l], vW[l]), (b[l], gb, mb[l], vb[l])):
            m1, v1 = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            w -= 1e-3 * (m1 / (1 - 0.9 ** step)) / (np.sqrt(v1 / (1 - 0.999 ** step)) + 1e-8)
    return dict(loss=float(np.mean(diff * diff)), W=W, b=b)
