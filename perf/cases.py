"""The calls whose speed is measured: what a user of gplite_gb300 has it do.

Every case goes through the public Python API on host arrays (the API's own
input form: R matrices, numpy arrays), so a pass includes the copies to and from
the device that such a call makes. The families:

  fit_predict   gp_fit, then gp_pred with variance at new inputs
  step          one step of a gradient optimiser: gp_fit(grad=True), energy and gradient
  predict       gp_pred with variance on a model that stays fitted
  classify      non-Gaussian likelihood (Laplace or EP), then gp_loo
  fitc          inducing-point fit of a large data set, then gp_pred
  batch         thousands of small regressions on a kept BatchPlan with new data
  served        a burst of mixed fit + predict requests to a running GPServer

Sizes are those of the benchmark configurations and of the tests, with ragged
ones between them.
"""
import math

import numpy as np
import torch

import gplite_gb300 as G
from gplite_gb300.batch import BatchPlan
from gplite_gb300.gp import model_field
from gplite_gb300.server import GPServer

JITTER = 1e-6
LOO_ORDER = 11


def listed():
    return [
        # the plain 1D regression of the first configuration: one energy evaluation of
        # gp_optim and its 300-point prediction; latency and launches are all of it
        dict(name="regression-200", family="fit_predict", precision="fp64", n=200, d=1, m=300, kernel="sexp",
             lscale=0.3, sigma=0.1),
        # one L-BFGS step on a data set of everyday size
        dict(name="step-1000", family="step", precision="fp64", n=1000, d=3, kernel="sexp+const", lscale=0.5,
             sigma=0.1),
        # the same at the size where the default precision still fits an interactive run
        dict(name="step-8192", family="step", precision="fp64", n=8192, d=8, kernel="matern52+const", lscale=0.7,
             sigma=0.05),
        # the large regression configuration: gp_energy and gradient in mixed precision
        dict(name="step-16384-mixed", family="step", precision="mixed", n=16384, d=8, kernel="matern52+const",
             lscale=0.7, sigma=0.05),
        # fit once, predict once, at a ragged size
        dict(name="regression-5003", family="fit_predict", precision="fp64", n=5003, d=4, m=1501,
             kernel="matern32", lscale=0.8, sigma=0.1),
        # the large regression's prediction: 8192 points on the resident model
        dict(name="predict-16384-mixed", family="predict", precision="mixed", n=16384, d=8, m=8192,
             kernel="matern52+const", lscale=0.7, sigma=0.05),
        # binary classification with Laplace and leave-one-out, default precision
        dict(name="laplace-3000", family="classify", precision="fp64", n=3000, d=4, lik="bernoulli",
             approx="laplace", lscale=0.5, magn=2.0),
        # the non-Gaussian configuration in mixed precision at its own size
        dict(name="laplace-8192-mixed", family="classify", precision="mixed", n=8192, d=4, lik="bernoulli",
             approx="laplace", lscale=0.5, magn=2.0),
        # the same model by expectation propagation
        dict(name="ep-2500", family="classify", precision="fp64", n=2500, d=4, lik="bernoulli", approx="ep",
             lscale=0.5, magn=2.0),
        # counts at 65536 points through 256 inducing inputs, 256 predictions (a served request's shape)
        dict(name="fitc-65536", family="fitc", precision="fp64", n=65536, d=4, m=256, inducing=256,
             lik="poisson", lscale=0.7, magn=0.7),
        # independent small regressions of uneven size, refitted with new data on a kept plan
        dict(name="batch-1024", family="batch", precision="mixed", count=1024, nmin=64, nmax=1024, m=128),
        # a burst of the served stream: sizes log-uniform, four of five requests Gaussian, one Poisson
        dict(name="served-32-mixed", family="served", precision="mixed", count=32, nmin=32, nmax=6000, m=256),
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    fam = rng.choice(["fit_predict", "fit_predict", "step", "step", "predict", "classify", "classify", "fitc", "batch",
                      "served"])
    prec = rng.choice(["fp64", "mixed"])
    top = 8192 if prec == "fp64" else 12000
    if fam == "fit_predict":
        return dict(family=fam, precision=prec, n=_logu(rng, 50, top * 3 // 4), d=rng.randint(1, 8), m=_logu(rng, 20, 2000),
                    kernel=rng.choice(["sexp", "matern32", "matern52+const"]), lscale=round(rng.uniform(0.3, 0.9), 3),
                    sigma=round(rng.uniform(0.05, 0.3), 3))
    if fam == "step":
        return dict(family=fam, precision=prec, n=_logu(rng, 100, top), d=rng.randint(1, 8),
                    kernel=rng.choice(["sexp+const", "matern32", "matern52+const"]),
                    lscale=round(rng.uniform(0.3, 0.9), 3), sigma=round(rng.uniform(0.05, 0.3), 3))
    if fam == "predict":
        return dict(family=fam, precision=prec, n=_logu(rng, 200, top * 3 // 4), d=rng.randint(2, 8),
                    m=_logu(rng, 50, 4000), kernel=rng.choice(["sexp", "matern52+const"]),
                    lscale=round(rng.uniform(0.4, 0.9), 3), sigma=round(rng.uniform(0.05, 0.3), 3))
    if fam == "classify":
        approx = rng.choice(["laplace", "ep"])
        return dict(family=fam, precision=prec, n=_logu(rng, 100, 3000 if approx == "ep" else 4500), d=rng.randint(2, 4),
                    lik=rng.choice(["bernoulli", "poisson"]) if approx == "laplace" else "bernoulli", approx=approx,
                    lscale=round(rng.uniform(0.4, 0.8), 3), magn=round(rng.uniform(0.6, 2.0), 3))
    if fam == "fitc":
        return dict(family=fam, precision="fp64", n=_logu(rng, 4000, 65536), d=4, m=_logu(rng, 50, 500),
                    inducing=rng.randint(64, 256), lik=rng.choice(["poisson", "gaussian"]),
                    lscale=round(rng.uniform(0.5, 0.8), 3), magn=0.7)
    if fam == "batch":
        return dict(family=fam, precision=prec, count=_logu(rng, 16, 1024 if prec == "mixed" else 256), nmin=64, nmax=1024,
                    m=128)
    return dict(family=fam, precision=prec, count=rng.randint(6, 32), nmin=32, nmax=_logu(rng, 500, 4000), m=256)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _latent(rng, x, lscale, magn, feats=64):
    """A random-Fourier-feature draw of a smooth GP with this lengthscale at the rows of x."""
    w = rng.standard_normal((x.shape[1], feats)) / lscale
    b = rng.uniform(0, 2 * math.pi, feats)
    a = rng.standard_normal(feats)
    return magn * math.sqrt(2.0 / feats) * (np.cos(x @ w + b) @ a)


def _problems(case, seed):
    """The small regressions: sizes and kernels from the plan's own seed (a plan is for fixed
    shapes), data from `seed`."""
    shape = np.random.default_rng(4)
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        n = int(round(math.exp(shape.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        d = int(shape.integers(1, 4))
        kind = "sexp" if shape.uniform() < 0.5 else "matern32"
        lscale = math.exp(shape.uniform(math.log(0.2), math.log(2.0)))
        sigma = shape.uniform(0.01, 0.3)
        x = rng.uniform(-2, 2, (n, d))
        y = _latent(rng, x, lscale, 1.0) + sigma * rng.standard_normal(n)
        out.append(dict(x=x, y=y, xt=rng.uniform(-2, 2, (case["m"], d)), kind=kind, lscale=lscale, magn=1.0,
                        sigma=sigma))
    return out


def _requests(case, seed):
    """The served burst: sizes and likelihoods from a seed of their own (as the kernels a
    service is set up with), data from `seed`; d = 2, sexp."""
    shape = np.random.default_rng(5)
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["count"]):
        n = int(round(math.exp(shape.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        c = dict(family="served", n=n, d=2, m=case["m"], kernel="sexp", lscale=round(shape.uniform(0.3, 1.0), 3),
                 lik="poisson" if i % 5 == 4 else "gaussian", sigma=0.1, magn=0.7 if i % 5 == 4 else 1.0)
        out.append((c, _data(c, int(rng.integers(1 << 40)))))
    return out


def _data(case, seed):
    rng = np.random.default_rng(seed)
    n, d, m = case["n"], case["d"], case.get("m", 0)
    if case["family"] in ("classify", "fitc") or d == 1:
        x, xt = rng.standard_normal((n, d)), rng.standard_normal((m, d))
    else:
        x, xt = rng.uniform(-1, 1, (n, d)), rng.uniform(-1, 1, (m, d))
    f = _latent(rng, x, case["lscale"], case.get("magn", 1.0))
    lik = case.get("lik", "gaussian")
    if lik == "bernoulli":
        y = (rng.uniform(size=n) < 1 / (1 + np.exp(-f))).astype(np.float64)
    elif lik == "poisson":
        y = rng.poisson(np.exp(np.minimum(f, 4.0))).astype(np.float64)
    else:
        y = f + case.get("sigma", 0.1) * rng.standard_normal(n)
    z = x[np.sort(rng.choice(n, case["inducing"], replace=False))] if "inducing" in case else None
    return x, y, xt, z


def _kernel_terms(case):
    """(kind, lscale, magn) per term."""
    return [("const", None, 1.0) if k == "const" else (k, case["lscale"], case.get("magn", 1.0))
            for k in case.get("kernel", "sexp").split("+")]


def _model(case, z):
    make = dict(sexp=G.cf_sexp, matern32=G.cf_matern32, matern52=G.cf_matern52)
    cfs = [G.cf_const(m) if k == "const" else make[k](lscale=ls, magn=m) for k, ls, m in _kernel_terms(case)]
    kind = case.get("lik", "gaussian")
    lik = (G.lik_gaussian(sigma=case.get("sigma", 0.1)) if kind == "gaussian"
           else G.lik_bernoulli() if kind == "bernoulli" else G.lik_poisson())
    method = (G.method_fitc(inducing=z) if z is not None
              else G.method_full())
    approx = G.approx_ep(damping=0.9) if case.get("approx") == "ep" else G.approx_laplace(tol=1e-6)
    return G.gp_init(cfs, lik, method, approx)


def prepare(case, seed):
    st = dict(case=case)
    if case["family"] == "batch":
        st["problems"] = _problems(case, seed)
        st["plan"] = BatchPlan(st["problems"], precision=case["precision"])
        st["plan"].run()  # the plan's one-off tuning and capture
        st["plan"].results()
        return st
    if case["family"] == "served":
        st["requests"] = [(_model(c, None), x, y, xt) for c, (x, y, xt, _) in _requests(case, seed)]
        st["server"] = GPServer(precision=case["precision"], workers=4)
        return st
    x, y, xt, z = _data(case, seed)
    st.update(x=x, y=y, xt=xt, gp=_model(case, z))
    if case["family"] == "predict":
        G.gp_fit(st["gp"], x, y, precision=case["precision"], grad=True)
    return st


def run(st):
    case = st["case"]
    fam, prec = case["family"], case["precision"]
    if fam == "batch":
        plan = st["plan"]
        plan.upload(st["problems"])
        plan.run()
        res = plan.results()
        return dict(log_evidence=np.array([r["log_evidence"] for r in res]),
                    mean=np.concatenate([r["mean"] for r in res]), var=np.concatenate([r["var"] for r in res]),
                    loos=np.concatenate([r["loos"] for r in res]))
    if fam == "served":
        srv = st["server"]
        res = [srv.poll(t) for t in [srv.submit(gp, x, y, xt=xt) for gp, x, y, xt in st["requests"]]]
        return dict(log_evidence=np.array([r["log_evidence"] for r in res]),
                    mean=np.concatenate([r["mean"] for r in res]), var=np.concatenate([r["var"] for r in res]))
    gp, x, y = st["gp"], st["x"], st["y"]
    if fam == "predict":
        p = G.gp_pred(gp, st["xt"], var=True)
        return dict(mean=p["mean"], var=p["var"])
    if fam == "step":
        G.gp_fit(gp, x, y, precision=prec, grad=True)
        return dict(energy=np.float64(G.gp_energy(gp)), grad=G.gp_energy_grad(gp))
    G.gp_fit(gp, x, y, precision=prec)
    if fam == "classify":
        loo = G.gp_loo(gp, x, y)
        return dict(energy=np.float64(G.gp_energy(gp)), fmean=model_field(gp, "fmean"), loos=loo["loos"])
    p = G.gp_pred(gp, st["xt"], var=True)
    return dict(energy=np.float64(G.gp_energy(gp)), mean=p["mean"], var=p["var"])


def work(case):
    """Inputs and outputs once, and the operations of the algorithm the result is defined by
    (a Cholesky factorisation is n^3/3, a triangular inverse n^3/3, a product 2 m n k)."""
    fam = case["family"]
    if fam == "batch":
        ns = [(len(p["y"]), p["x"].shape[1]) for p in _problems(case, 0)]
        m = case["m"]
        return dict(bytes=8.0 * sum(n * (d + 2) + m * (d + 2) + 1 for n, d in ns),
                    flops=float(sum(2 * n ** 3 / 3 + n * n * (m + 1.5 * d + 10) for n, d in ns)))
    if fam == "served":
        shapes = [(c["n"], c["lik"]) for c, _ in _requests(case, 0)]
        m = case["m"]
        return dict(bytes=8.0 * sum(4 * n + 4 * m for n, _ in shapes),
                    flops=float(sum((6 if k == "poisson" else 1) * n ** 3 / 3 + n * n * (m + 11) for n, k in shapes)))
    n, d, m = case["n"], case["d"], case.get("m", 0)
    io = 8.0 * (n * (d + 1) + m * (d + 2) + 8)
    cov = n * n / 2 * (3 * d + 15)
    if fam == "fit_predict":
        return dict(bytes=io, flops=cov + n ** 3 / 3 + float(n) * n * m + n * m * (3 * d + 15))
    if fam == "step":
        return dict(bytes=io, flops=1.5 * cov + float(n) ** 3)
    if fam == "predict":
        return dict(bytes=8.0 * (m * (d + 2) + n * n / 2), flops=float(n) * n * m + n * m * (3 * d + 15))
    if fam == "classify":
        sweeps = 6
        each = n ** 3 / 3 * (2 if case["approx"] == "ep" else 1)
        return dict(bytes=io + 16.0 * n, flops=cov + sweeps * each + n ** 3 / 3)
    k = case["inducing"]
    sweeps = 1 if case.get("lik", "gaussian") == "gaussian" else 8
    return dict(bytes=io, flops=float(n) * k * (3 * d + 15) + float(n) * k * k * (1 + sweeps) + sweeps * k ** 3 / 3)


# ---------------------------------------------------------------------------
# the same results in 64 bits with torch
# ---------------------------------------------------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _r2(a, b):
    out = torch.zeros(a.shape[0], b.shape[0], dtype=torch.float64, device=a.device)
    for j in range(a.shape[1]):
        out.add_((a[:, j:j + 1] - b[:, j][None, :]).square_())
    return out


def _cov(terms, a, b):
    K = torch.zeros(a.shape[0], b.shape[0], dtype=torch.float64, device=a.device)
    r2 = _r2(a, b)
    for k, ls, m in terms:
        if k == "const":
            K += m * m
        elif k == "sexp":
            K += m * m * torch.exp(-0.5 * r2 / (ls * ls))
        else:
            u = torch.sqrt(r2) * (math.sqrt(3.0 if k == "matern32" else 5.0) / ls)
            K += m * m * (1 + u if k == "matern32" else 1 + u + u * u / 3) * torch.exp(-u)
    return K


def _dcov(terms, a):
    """dK/dlog(parameter) in get_param order: lscale, magn per term."""
    r2 = _r2(a, a)
    for k, ls, m in terms:
        if k == "const":
            yield torch.full_like(r2, 2 * m * m)
            continue
        if k == "sexp":
            e = m * m * torch.exp(-0.5 * r2 / (ls * ls))
            yield e * r2 / (ls * ls)
            yield 2 * e
            continue
        u = torch.sqrt(r2) * (math.sqrt(3.0 if k == "matern32" else 5.0) / ls)
        e = m * m * torch.exp(-u)
        if k == "matern32":
            yield e * u * u
            yield 2 * (1 + u) * e
        else:
            yield e * u * u * (1 + u) / 3
            yield 2 * (1 + u + u * u / 3) * e


def _tri(L, b, trans=False):
    v = b.reshape(b.shape[0], -1)
    r = torch.linalg.solve_triangular(L.T if trans else L, v, upper=trans)
    return r.reshape(b.shape)


def _loglik(lik, f, y, sigma=0.0):
    if lik == "gaussian":
        return -math.log(sigma) - 0.5 * math.log(2 * math.pi) - 0.5 * ((y - f) / sigma) ** 2
    if lik == "bernoulli":
        return y * torch.nn.functional.logsigmoid(f) + (1 - y) * torch.nn.functional.logsigmoid(-f)
    return y * f - torch.exp(f) - torch.lgamma(y + 1)


def _gradlik(lik, f, y):
    if lik == "bernoulli":
        mu = 1 / (1 + torch.exp(-f))
        return mu * (1 - mu) * (y / mu - (1 - y) / (1 - mu))
    mu = torch.exp(f)
    return (y / mu - 1) * mu


def _pseudo(lik, f, y, sigma):
    """Laplace pseudo-data: the curvature is the forward difference the method is defined with."""
    if lik == "gaussian":
        return y.clone(), torch.full_like(y, sigma * sigma)
    g = _gradlik(lik, f, y)
    g2 = (_gradlik(lik, f + 1e-6, y) - g) / 1e-6
    g2 = torch.sign(g2) * torch.clamp(g2.abs(), min=1e-12)
    return f - g / g2, -1 / g2


def _gh(p, dev):
    """Nodes and weights of the standard normal's Gauss-Hermite rule."""
    x, w = np.polynomial.hermite_e.hermegauss(p)
    t = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
    return t(x), t(w / w.sum())


def _loos(lik, mean, var, y, sigma):
    x, w = _gh(LOO_ORDER, mean.device)
    ll = _loglik(lik, mean[:, None] + torch.sqrt(var)[:, None] * x[None, :], y[:, None], sigma)
    return torch.logsumexp(ll + torch.log(w)[None, :], 1)


def _factor(K, V):
    s = torch.sqrt(1 / V)
    B = s[:, None] * K * s[None, :]
    B.diagonal().add_(1.0)
    return s, torch.linalg.cholesky(B)


def _laplace(case, K, y, sigma=0.0):
    """Newton iteration from f = 0 on B = I + V^-1/2 K V^-1/2."""
    lik = case.get("lik", "gaussian")
    f = torch.zeros_like(y)
    for _ in range(1 if lik == "gaussian" else 30):
        z, V = _pseudo(lik, f, y, sigma)
        s, L = _factor(K, V)
        alpha = s * _tri(L, _tri(L, s * z), True)
        new = K @ alpha
        diff = (new - f).abs().max()
        f = new
        if diff < 1e-6:
            break
    lml = _loglik(lik, f, y, sigma).sum() - 0.5 * (f @ alpha) - torch.log(L.diagonal()).sum()
    return dict(lml=lml, f=f, alpha=alpha, z=z, V=V, s=s, L=L)


def _laplace_loo(case, r, y, sigma=0.0):
    n = y.shape[0]
    W = _tri(r["L"], torch.eye(n, dtype=torch.float64, device=y.device))
    D = r["V"] + JITTER
    pv = D - D * D * ((W * W).sum(0) / r["V"])
    lv = 1 / (1 / pv - 1 / r["V"])
    return _loos(case.get("lik", "gaussian"), r["f"] - lv * (r["z"] - r["f"]) / r["V"], lv, y, sigma)


def _ep(case, K, y):
    """Parallel EP with the damping schedule it is defined by."""
    lik, n = case["lik"], y.shape[0]
    x, w = _gh(11, y.device)
    P, z, f, fv = torch.zeros_like(y), torch.zeros_like(y), torch.zeros_like(y), K.diagonal().clone()
    eye = torch.eye(n, dtype=torch.float64, device=y.device)
    damp, old = 0.9, math.inf
    for _ in range(100):
        cp = 1 / fv - P
        cm, cv = (f / fv - z * P) / cp, 1 / cp
        g = cm[:, None] + torch.sqrt(cv)[:, None] * x[None, :]
        ll = _loglik(lik, g, y[:, None])
        logC = torch.logsumexp(ll + torch.log(w)[None, :], 1)
        q = torch.exp(ll - logC[:, None]) * w[None, :]
        mt = (g * q).sum(1)
        vt = ((g - mt[:, None]) ** 2 * q).sum(1)
        Pn = damp * (1 / vt - 1 / cv) + (1 - damp) * P
        zn = (damp * (mt / vt - cm / cv) + (1 - damp) * z * P) / Pn
        V = 1 / Pn
        if not bool((V > 0).all()):
            return None
        s, L = _factor(K, V)
        alpha = s * _tri(L, _tri(L, s * zn), True)
        new = K @ alpha
        Wi = _tri(L, eye)
        fvn = V * (1 - (Wi * Wi).sum(0))
        lml = (-torch.log(L.diagonal()).sum() - 0.5 * torch.log(V).sum() - 0.5 * (zn @ alpha) + logC.sum()
               + 0.5 * torch.log(cv + V).sum() + 0.5 * ((cm - zn) ** 2 / (cv + V)).sum())
        diff = float((new - f).abs().max())
        if diff > old:
            damp *= 0.9
            continue
        damp = max(damp, 0.1)
        f, fv, z, P, old = new, fvn, zn, Pn, diff
        if diff < 1e-4:
            break
    return dict(lml=lml, f=new, loos=_loos(lik, cm, cv, y, 0.0))


def _fitc(case, x, y, xt, z, sigma):
    lik, terms = case["lik"], _kernel_terms(case)
    Kz = _cov(terms, z, z)
    Kz.diagonal().add_(JITTER)
    Kxz = _cov(terms, x, z)
    Lz = torch.linalg.cholesky(Kz)
    kd = sum(m * m for _, _, m in terms)
    A = _tri(Lz, Kxz.T.contiguous())
    D = kd + JITTER - (A * A).sum(0)
    f, old = torch.zeros_like(y), -math.inf
    for _ in range(1 if lik == "gaussian" else 30):
        zz, V = _pseudo(lik, f, y, sigma)
        S = D + V
        U = Kxz / S[:, None]
        Ls = torch.linalg.cholesky(Kz + Kxz.T @ U)
        alpha = zz / S - U @ _tri(Ls, _tri(Ls, U.T @ zz), True)
        f = Kxz @ _tri(Lz, _tri(Lz, Kxz.T @ alpha), True) + D * alpha
        logdet = torch.log(S).sum() - 2 * torch.log(Lz.diagonal()).sum() + 2 * torch.log(Ls.diagonal()).sum()
        lpu = float(_loglik(lik, f, y, sigma).sum() - 0.5 * (f @ alpha))
        if abs(lpu - old) < 1e-6:
            break
        old = lpu
    lml = _loglik(lik, f, y, sigma).sum() - 0.5 * (f @ alpha) + 0.5 * (torch.log(V).sum() - logdet)
    A2 = _tri(Lz, _cov(terms, xt, z).T.contiguous())
    mean = A2.T @ (A @ alpha)
    G1 = _tri(Ls, U.T @ A.T)
    red = (A / S[None, :]) @ A.T - G1.T @ G1  # A C^-1 A^T
    var = (A2 * A2).sum(0) + (kd - (A2 * A2).sum(0)) - (A2 * (red @ A2)).sum(0)
    return lml, mean, var


def exact(case, seed):
    dev = _dev()
    t = lambda a: None if a is None else torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    h = lambda a: a.cpu().numpy()  # noqa: E731
    if case["family"] == "batch":
        out = dict(log_evidence=[], mean=[], var=[], loos=[])
        for p in _problems(case, seed):
            x, y, xt, terms = t(p["x"]), t(p["y"]), t(p["xt"]), [(p["kind"], p["lscale"], p["magn"])]
            K = _cov(terms, x, x)
            K.diagonal().add_(JITTER)
            r = _laplace({}, K, y, p["sigma"])
            Kt = _cov(terms, x, xt)
            a = _tri(r["L"], r["s"][:, None] * Kt)
            out["log_evidence"].append(r["lml"])
            out["mean"].append(Kt.T @ r["alpha"])
            out["var"].append(p["magn"] ** 2 - (a * a).sum(0))
            out["loos"].append(_laplace_loo({}, r, y, p["sigma"]))
        return dict(log_evidence=h(torch.stack(out["log_evidence"])), mean=h(torch.cat(out["mean"])),
                    var=h(torch.cat(out["var"])), loos=h(torch.cat(out["loos"])))
    if case["family"] == "served":
        parts = []
        for c, (x, y, xt, _) in _requests(case, seed):
            x, y, xt = t(x), t(y), t(xt)
            K = _cov(_kernel_terms(c), x, x)
            K.diagonal().add_(JITTER)
            r = _laplace(c, K, y, c["sigma"])
            Kt = _cov(_kernel_terms(c), x, xt)
            a = _tri(r["L"], r["s"][:, None] * Kt)
            parts.append((r["lml"], Kt.T @ r["alpha"], c["magn"] ** 2 - (a * a).sum(0)))
        lml, mean, var = zip(*parts)
        return dict(log_evidence=h(torch.stack(lml)), mean=h(torch.cat(mean)), var=h(torch.cat(var)))
    x, y, xt, z = (t(a) for a in _data(case, seed))
    sigma, terms = case.get("sigma", 0.1), _kernel_terms(case)
    en = lambda v: np.float64(-float(v))  # noqa: E731  (the default priors are flat)
    if case["family"] == "fitc":
        lml, mean, var = _fitc(case, x, y, xt, z, sigma)
        return dict(energy=en(lml), mean=h(mean), var=h(var))
    K = _cov(terms, x, x)
    K.diagonal().add_(JITTER)
    if case["family"] == "classify":
        if case["approx"] == "ep":
            r = _ep(case, K, y)
            return None if r is None else dict(energy=en(r["lml"]), fmean=h(r["f"]), loos=h(r["loos"]))
        r = _laplace(case, K, y)
        return dict(energy=en(r["lml"]), fmean=h(r["f"]), loos=h(_laplace_loo(case, r, y)))
    r = _laplace(case, K, y, sigma)
    if case["family"] == "step":
        del K
        C = torch.cholesky_inverse(r["L"])
        C.mul_(-1 / (sigma * sigma)).addr_(r["alpha"], r["alpha"])  # alpha alpha^T - C^-1
        g = [float(-0.5 * (C * dK).sum()) for dK in _dcov(terms, x)]
        g.append(float(-sigma * sigma * C.diagonal().sum()))
        return dict(energy=en(r["lml"]), grad=np.array(g))
    Kt = _cov(terms, x, xt)
    mean = Kt.T @ r["alpha"]
    a = _tri(r["L"], Kt * r["s"][:, None])
    var = sum(m * m for _, _, m in terms) - (a * a).sum(0)
    return (dict(mean=h(mean), var=h(var)) if case["family"] == "predict"
            else dict(energy=en(r["lml"]), mean=h(mean), var=h(var)))
