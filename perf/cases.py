"""What a user of the TLR log-likelihood has it do, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` makes the inputs a user's program holds before the
call, `run` is one call through the package's public entry points, `work` the bytes and operations
that call cannot do without, and `exact` its result from plain NumPy in 64 bits (where that takes
seconds only).  `listed` are the named cases, `draw` gives more of the same ranges.

Sites are uniform on the unit square, observations a Matern field plus nugget noise from random
Fourier features (the spectral density of the Matern kernel), so that no dense factor is needed.
"""
import math

import numpy as np
import torch

import adaptive_tlr_pilots_b200 as tlr

MEAN_RANK = 5.0  # typical factor rank at tau = 0.9 (4.6 at N = 50,000), for work()


def listed():
    base = dict(sigma2=1.0, range=0.3, eta=0.05, nu=1.5, rule="adaptive", value=0.9)
    return [
        # the smallest fits: an optimizer's calls on a thousand sites, latency and launches count;
        # the form that takes unordered sites (Morton order inside the call)
        dict(base, name="loglik_n1030_b100", family="loglik", form="locs", n=1030, b=100),
        # one objective evaluation of the pilot scripts' fits, Morton-ordered host arrays
        dict(base, name="loglik_n4000_b250", family="loglik", form="dropin", n=4000, b=250),
        # the regime sweeps: Matern 5/2, a tighter budget, a last tile of seven sites
        dict(base, name="loglik_n10007_b250", family="loglik", form="locs", n=10007, b=250, nu=2.5, value=0.5),
        # the N = 20,000 sweep at its rough corner (short range, small nugget: higher ranks)
        dict(base, name="loglik_n20000_b500", family="loglik", form="dropin", n=20000, b=500, range=0.1, eta=0.005),
        # the tile size of the largest fields
        dict(base, name="loglik_n12000_b1000", family="loglik", form="dropin", n=12000, b=1000, range=1.0),
        # value and gradient for a quasi-Newton fit, every step in 64 bits, odd tile size
        dict(base, name="grad_n4000_b203", family="grad", form="dropin", n=4000, b=203),
        # the same at the headline size
        dict(base, name="grad_n50000_b500", family="grad", form="dropin", n=50000, b=500),
        # torch optimizer over FP32 parameters through autograd, mixed precision
        dict(base, name="autograd_n20000_b500", family="grad", form="autograd", n=20000, b=500, range=0.2),
        # one iteration of four chains from host data: the headline workload, mixed precision, batched
        dict(base, name="batch4_n50000_b500", family="batch", n=50000, b=500, count=4),
        # kriging at the 300 held-out sites with the factor of the fitted parameters
        dict(base, name="predict_n20000_m300", family="predict", n=20000, b=500, m=300),
        # assembled-matrix rule: the covariance with every off-diagonal tile truncated, fixed rule
        dict(base, name="cov_n8000_b250", family="cov", n=8000, b=250, rule="fixed", value=1e-5),
        # data loading: Z-order permutation of the sites
        dict(name="morton_n50000", family="morton", n=50000),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any family, sizes spread over the listed range (logarithmically), odd tile
    sizes and ragged last tiles among them, at most the cost of the largest listed case."""
    family = rng.choice(["loglik", "loglik", "loglik", "grad", "grad", "batch", "predict", "cov", "morton"])
    if family == "morton":
        return dict(family=family, n=_logint(rng, 1000, 1000000))
    top = dict(loglik=30000, grad=24000, batch=16000, predict=20000, cov=9000)[family]
    n = _logint(rng, 1000, top)
    lo = max(64, -(-n // 80))
    b = _logint(rng, lo, max(lo + 1, min(1000, n // 4)))
    if rng.random() < 0.5:
        b = max(lo, b // 10 * 10)
    if b in (319, 320):  # tile sizes the compression cannot be launched at
        b = 321
    c = dict(family=family, n=n, b=b, sigma2=round(rng.uniform(0.5, 2.0), 3),
             range=round(math.exp(rng.uniform(math.log(0.1), math.log(1.0))), 4),
             eta=round(math.exp(rng.uniform(math.log(0.005), math.log(0.1))), 5), nu=rng.choice([1.5, 1.5, 2.5]),
             rule="adaptive", value=round(rng.uniform(0.3, 0.95), 3))
    if family in ("loglik", "cov") and rng.random() < 0.3:  # the fixed relative rule
        c.update(rule="fixed", value=float("%.3g" % math.exp(rng.uniform(math.log(1e-6), math.log(3e-5)))),
                 eta=max(c["eta"], 0.03))
    if family == "loglik":
        c["form"] = rng.choice(["locs", "dropin"])
    elif family == "grad":
        c["form"] = rng.choice(["dropin", "dropin", "autograd"])
    elif family == "batch":
        c["count"] = rng.randint(2, 6)
    elif family == "predict":
        c["m"] = _logint(rng, 1, 1000)
    return c


# ---------------------------------------------------------------------------------- inputs
def _morton(xy, order=10):
    """Z-order permutation, ties in input order."""
    side = 1 << order
    q = np.clip((xy * side).astype(np.int64), 0, side - 1)
    key = np.zeros(len(xy), dtype=np.int64)
    for bit in range(order):
        key |= ((q[:, 0] >> bit) & 1) << (2 * bit)
        key |= ((q[:, 1] >> bit) & 1) << (2 * bit + 1)
    return np.argsort(key, kind="stable")


def _theta(c):
    return (c["sigma2"], c["range"], c["eta"])


def _sites(c, seed):
    """(S, y): n sites in random order and a field with the case's parameters at them."""
    rng = np.random.default_rng(seed)
    n, nu, terms = c["n"], c["nu"], 512
    S = rng.random((n, 2))
    # frequencies of the Matern kernel's spectral density in the plane: a bivariate t
    w = rng.standard_normal((terms, 2)) * np.sqrt(2 * nu / rng.chisquare(2 * nu, terms))[:, None] / c["range"]
    phase = rng.uniform(0, 2 * np.pi, terms)
    noise = rng.standard_normal(n)
    with torch.no_grad():
        f = torch.from_numpy(S).cuda() @ torch.from_numpy(w.T.copy()).cuda() + torch.from_numpy(phase).cuda()
        f = torch.cos(f).sum(1).cpu().numpy()
    y = math.sqrt(2 * c["sigma2"] / terms) * f + math.sqrt(c["sigma2"] * c["eta"]) * noise
    return S, y


def _ordered(c, seed):
    S, y = _sites(c, seed)
    p = _morton(S)
    return np.ascontiguousarray(S[p]), np.ascontiguousarray(y[p])


def _held_out(c, seed):
    return np.random.default_rng(seed + 7919).random((c["m"], 2))


def _chain_thetas(c, seed):
    """Parameter vectors of chains near the mode: theta exp(0.05 z)."""
    z = np.random.default_rng(seed + 104729).standard_normal((c["count"], 3))
    return np.array(_theta(c)) * np.exp(0.05 * z)


_BATCH = {}


def _workspaces(c):
    """The sampler's workspaces, kept while its problem size stays."""
    key = (c["n"], c["b"], c["count"])
    if key not in _BATCH:
        for old in _BATCH.values():
            old.close()
        _BATCH.clear()
        _BATCH[key] = tlr.PlanBatch(*key, precision="mixed")
    return _BATCH[key]


def prepare(case, seed):
    c = case
    f = c["family"]
    if f == "morton":
        return dict(c=c, xy=np.random.default_rng(seed).random((c["n"], 2)))
    if f == "loglik" and c["form"] == "locs":
        S, y = _sites(c, seed)
        return dict(c=c, S=S, y=y)
    S, y = _ordered(c, seed)
    st = dict(c=c, S=S, y=y, bounds=tlr.tile_bounds(c["n"], c["b"]))
    if f == "batch":
        st["batch"] = _workspaces(c)
        st["thetas"] = _chain_thetas(c, seed)
    elif f == "predict" or (f == "grad" and c["form"] == "autograd"):
        plan = tlr.Plan(c["n"], c["b"])
        plan.set_kernel(c["nu"])
        plan.set_data(S, y)
        st["plan"] = plan
        if f == "predict":
            plan.evaluate(_theta(c), c["rule"], c["value"])
            st["factor"] = tlr.TLRFactor(plan)
            st["Sp"] = _held_out(c, seed)
        else:
            plan.set_precision("mixed")
            st["theta"] = torch.tensor(_theta(c), dtype=torch.float32, requires_grad=True)
    return st


# ---------------------------------------------------------------------------------- one call
def _f64(v):
    """A 64-bit result as an array value: it stays 64 bits wherever it is kept."""
    return None if v is None else np.float64(v)


_INFO = ("stored_sigma", "max_rank_sigma", "stored_factor", "max_rank_factor")


def _numbers(info):
    return {k: info[k] for k in _INFO if k in info}


def run(st):
    c = st["c"]
    f = c["family"]
    if f == "morton":
        return tlr.morton_order(st["xy"])
    theta, rule, value = _theta(c), c["rule"], c["value"]
    tlr.set_kernel(c["nu"])
    if f == "loglik" and c["form"] == "locs":
        key = {"tau": value} if rule == "adaptive" else {"eps": value}
        ll, ranks, pd = tlr.loglik(theta, st["S"], st["y"], c["b"], rule, **key)
        return dict(ll=_f64(ll), ranks=ranks, pd=pd)
    if f == "loglik":
        ll, _, info = tlr.tlr_loglik(st["S"], st["y"], theta, st["bounds"], rule, value)
        return dict(ll=_f64(ll), logdet=_f64(info.get("logdet")), quad=_f64(info.get("quad")), info=_numbers(info))
    if f == "grad" and c["form"] == "dropin":
        ll, g, info = tlr.tlr_loglik_grad(st["S"], st["y"], theta, st["bounds"], rule, value)
        return dict(ll=_f64(ll), grad=g, logdet=_f64(info.get("logdet")), quad=_f64(info.get("quad")),
                    info=_numbers(info))
    if f == "grad":
        th = st["theta"]
        th.grad = None
        ll = tlr.TLRLogLik.apply(th, st["plan"], rule, value)
        ll.backward()
        return dict(ll=ll.detach(), grad=th.grad)
    if f == "batch":
        st["batch"].set_data(st["S"], st["y"])
        got = st["batch"].evaluate(st["thetas"], rule, value)
        # the chains keep the mixed path's gradients (FP32 products) in FP32
        grads = [None if g is None else g.astype(np.float32) for _, g, _ in got]
        return dict(ll=[_f64(ll) for ll, _, _ in got], grad=grads, status=[s for _, _, s in got])
    if f == "predict":
        mu, sd = tlr.tlr_predict(st["S"], st["y"], st["Sp"], theta, st["bounds"], st["factor"])
        return dict(mu=mu, sd=sd)
    K, info = tlr.make_cov(st["S"], theta, rule, value, st["bounds"])
    return dict(K=K, stored=info[0], max_rel=info[1], max_abs=info[2], fro=info[3], ranks=np.array(info[4]))


def work(case):
    """Inputs read once, outputs written once; the covariance evaluated once per pair of sites (20
    operations) with one product of each entry with a factor, the diagonal Cholesky, the panel
    solves, one product per trailing pair and the dense blocks of the selected inversion, at the
    factor's typical rank."""
    c = case
    n = c["n"]
    if c["family"] == "morton":
        return {"bytes": 16.0 * n + 8.0 * n, "flops": 0.0}
    b, r = c["b"], MEAN_RANK
    nB = -(-n // b)
    tiles, pairs = nB * (nB - 1) / 2, nB * (nB - 1) * (nB - 2) / 6
    compress = n * n / 2.0 * (20 + 2 * r)
    factor = nB * b ** 3 / 3.0 + tiles * (b * b * r + 4 * b * r * r) + pairs * (4 * b * r * r + 8 * b * 4 * r * r)
    back = sum((nB - m) * (2.0 * b * b * r * (nB - m) + 2.0 * b * b * r * m * 2) for m in range(nB)) + n * n / 2.0 * 25
    data = 24.0 * n
    if c["family"] == "loglik":
        return {"bytes": data + 4 * tiles + 32, "flops": compress + factor}
    if c["family"] == "grad":
        return {"bytes": data + 64, "flops": compress + factor + back}
    if c["family"] == "batch":
        return {"bytes": data + 64 * c["count"], "flops": c["count"] * (compress + factor + back)}
    if c["family"] == "predict":
        stored = 8.0 * (nB * b * b / 2.0 + tiles * 2 * b * r)
        return {"bytes": stored + data + 32.0 * c["m"], "flops": (c["m"] + 2.0) * (n * b + 4.0 * tiles * b * r)}
    return {"bytes": data + 8.0 * n * n, "flops": compress}


# ---------------------------------------------------------------------------------- plain NumPy
def _cov(A, B, c):
    h = np.sqrt((A[:, None, 0] - B[None, :, 0]) ** 2 + (A[:, None, 1] - B[None, :, 1]) ** 2)
    x = math.sqrt(2 * c["nu"]) * h / c["range"]
    poly = 1 + x + x * x / 3 if c["nu"] == 2.5 else 1 + x
    return c["sigma2"] * poly * np.exp(-x)


def _dcov_drange(A, B, c):
    h = np.sqrt((A[:, None, 0] - B[None, :, 0]) ** 2 + (A[:, None, 1] - B[None, :, 1]) ** 2)
    x = math.sqrt(2 * c["nu"]) * h / c["range"]
    poly = x * x * (1 + x) / 3 if c["nu"] == 2.5 else x * x
    return c["sigma2"] * poly * np.exp(-x) / c["range"]


def _rank(s, c, fro, b):
    """Smallest r whose tail sqrt(sum_{t>=r} s_t^2) meets the rule."""
    limit = c["value"] * fro if c["rule"] == "fixed" else c["value"] * b * c["sigma2"] * c["eta"] / c["n"]
    tail = np.append(np.sqrt(np.cumsum(s[::-1] ** 2)[::-1]), 0.0)
    return int(np.argmax(tail <= limit)), tail


def _truncate(T, c, b):
    u, s, vt = np.linalg.svd(T, full_matrices=False)
    r, tail = _rank(s, c, float(np.linalg.norm(s)), b)
    return u[:, :r] * s[:r], vt[:r].T, tail[r], tail[0]


def _factor(S, c):
    """(diagonal tiles, {(i, k): (U, V)}) of the right-looking TLR Cholesky; None if not PD."""
    n = c["n"]
    edges = list(range(0, n, c["b"])) + [n]
    nB, b = len(edges) - 1, edges[1]
    X = [S[edges[t]:edges[t + 1]] for t in range(nB)]
    D, off = [], {}
    for i in range(nB):
        A = _cov(X[i], X[i], c)
        A[np.diag_indices_from(A)] += c["sigma2"] * c["eta"]
        D.append(A)
        for j in range(i):
            off[i, j] = _truncate(_cov(X[i], X[j], c), c, b)[:2]
    for k in range(nB):
        try:
            D[k] = np.linalg.cholesky(D[k])
        except np.linalg.LinAlgError:
            return None
        for i in range(k + 1, nB):
            U, V = off[i, k]
            off[i, k] = (U, np.linalg.solve(D[k], V))
        for i in range(k + 1, nB):
            Ui, Vi = off[i, k]
            if not Ui.shape[1]:
                continue
            D[i] = D[i] - Ui @ (Vi.T @ Vi) @ Ui.T
            for j in range(k + 1, i):
                Uj, Vj = off[j, k]
                if not Uj.shape[1]:
                    continue
                U, V = np.hstack([off[i, j][0], -Ui @ (Vi.T @ Vj)]), np.hstack([off[i, j][1], Uj])
                qu, ru = np.linalg.qr(U)
                qv, rv = np.linalg.qr(V)
                u, s, vt = np.linalg.svd(ru @ rv.T)
                r = _rank(s, c, float(np.linalg.norm(s)), b)[0]
                off[i, j] = (qu @ (u[:, :r] * s[:r]), qv @ vt[:r].T)
    return edges, D, off


def _forward(fac, B):
    """L^{-1} B."""
    edges, D, off = fac
    Z = np.array(B, dtype=np.float64)
    for k in range(len(D)):
        a, e = edges[k], edges[k + 1]
        Z[a:e] = np.linalg.solve(D[k], Z[a:e])
        for i in range(k + 1, len(D)):
            U, V = off[i, k]
            Z[edges[i]:edges[i + 1]] -= U @ (V.T @ Z[a:e])
    return Z


def _backward(fac, Z):
    """L^{-T} Z."""
    edges, D, off = fac
    X = np.array(Z, dtype=np.float64)
    for k in range(len(D) - 1, -1, -1):
        a, e = edges[k], edges[k + 1]
        for i in range(k + 1, len(D)):
            U, V = off[i, k]
            X[a:e] -= V @ (U.T @ X[edges[i]:edges[i + 1]])
        X[a:e] = np.linalg.solve(D[k].T, X[a:e])
    return X


def _seconds(c):
    """About how long the factorization takes in NumPy."""
    b = c["b"]
    nB = -(-c["n"] // b)
    return nB * nB / 2 * b ** 3 * 1.2e-9 + nB ** 3 / 6 * (8e-4 + 1.5e-6 * b)


def _exact_loglik(S, y, c):
    fac = _factor(S, c)
    if fac is None:
        return None
    z = _forward(fac, y)
    logdet, quad = 2 * sum(float(np.log(np.diag(d)).sum()) for d in fac[1]), float(z @ z)
    return fac, -0.5 * (quad + logdet + c["n"] * math.log(2 * math.pi)), logdet, quad


def _exact_grad(S, y, c):
    got = _exact_loglik(S, y, c)
    if got is None:
        return None
    fac, ll, logdet, quad = got
    n = c["n"]
    Li = _forward(fac, np.eye(n))
    alpha = Li.T @ (Li @ y)
    W = 0.5 * (np.outer(alpha, alpha) - Li.T @ Li)  # d loglik / d Sigma with the ranks frozen
    g = [float((_cov(S, S, c) * W).sum()) / c["sigma2"] + c["eta"] * float(np.trace(W)),
         float((_dcov_drange(S, S, c) * W).sum()), c["sigma2"] * float(np.trace(W))]
    return ll, np.array(g), logdet, quad


def exact(case, seed):
    c = case
    f = c["family"]
    if f == "morton":
        return _morton(np.random.default_rng(seed).random((c["n"], 2)))
    if f == "cov":
        b = c["b"]
        nB = -(-c["n"] // b)
        if nB * nB / 2 * b ** 3 * 1.2e-9 > 12:
            return None
        S, _ = _ordered(c, seed)
        K = _cov(S, S, c)
        K[np.diag_indices_from(K)] += c["sigma2"] * c["eta"]
        rel, worst, fro2 = 0.0, 0.0, 0.0
        edges = list(range(0, c["n"], b)) + [c["n"]]
        for i in range(nB):
            for j in range(i):
                a, e, g, h = edges[i], edges[i + 1], edges[j], edges[j + 1]
                U, V, tail, norm = _truncate(K[a:e, g:h], c, b)
                K[a:e, g:h] = U @ V.T
                K[g:h, a:e] = K[a:e, g:h].T
                rel, worst, fro2 = max(rel, tail / norm), max(worst, tail), fro2 + 2 * tail * tail
        return dict(K=K, stored=None, max_rel=rel, max_abs=worst, fro=math.sqrt(fro2), ranks=None)
    if _seconds(c) > 12 or (f in ("grad", "batch") and c["n"] > 5000):
        return None
    if f == "loglik":
        S, y = _sites(c, seed)
        p = _morton(S)
        got = _exact_loglik(S[p], y[p], c)
        if got is None:
            return None
        if c["form"] == "locs":
            return dict(ll=_f64(got[1]), ranks=None, pd=None)
        return dict(ll=_f64(got[1]), logdet=_f64(got[2]), quad=_f64(got[3]), info=None)
    S, y = _ordered(c, seed)
    if f == "grad":
        if c["form"] == "autograd":  # the parameters as the call sees them
            s2, rg, eta = (float(v) for v in np.array(_theta(c), dtype=np.float32))
            c = dict(c, sigma2=s2, range=rg, eta=eta)
        got = _exact_grad(S, y, c)
        if got is None:
            return None
        if c["form"] == "autograd":
            return dict(ll=_f64(got[0]), grad=got[1].astype(np.float32))
        return dict(ll=_f64(got[0]), grad=got[1], logdet=_f64(got[2]), quad=_f64(got[3]), info=None)
    if f == "batch":
        if c["count"] * _seconds(c) > 12:
            return None
        each = []
        for t in _chain_thetas(c, seed):
            got = _exact_grad(S, y, dict(c, sigma2=float(t[0]), range=float(t[1]), eta=float(t[2])))
            if got is None:
                return None
            each.append(got)
        return dict(ll=[_f64(g[0]) for g in each], grad=[g[1].astype(np.float32) for g in each], status=None)
    fac = _factor(S, c)
    if fac is None:
        return None
    Kp = _cov(_held_out(c, seed), S, c)
    mu = Kp @ _backward(fac, _forward(fac, y))
    Wp = _forward(fac, Kp.T)
    var = c["sigma2"] * (1 + c["eta"]) - (Wp * Wp).sum(0)
    return dict(mu=mu, sd=np.sqrt(np.clip(var, 1e-12, None)))
