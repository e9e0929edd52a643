"""Workloads of the framework's public entry points, for timing and comparison.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges,
``prepare`` makes a case's inputs, ``run`` is one pass as a user's program
makes it, ``work`` the bytes and operations that pass cannot do without and
``exact`` its results in 64-bit arithmetic without the framework.

Counts are negative binomial with Var = mu + theta mu^2 over the designs of
``devil_b200.synthetic`` (intercept + condition, plus one-hot cell types or
N(0, 1) covariates), gene means and dispersions log-normal as there.  Genes
seen in well under one cell in a hundred, or with fewer than a few dozen
counts expected in a cell type, are left out, as users filter them, and one
gene is present in every cell (cells without counts are filtered too).
"""
import ctypes as C
import math

import numpy as np
import torch

import devil_b200 as dv
from devil_b200 import _lib as L

# location and spread of the log gene means, by design
_MEANS = {"binary": (-3.0, 1.5), "types": (-3.8, 2.0), "patients": (-3.0, 1.5), "continuous": (-2.0, 1.0),
          "pilot": (0.0, 1.5)}


def listed():
    return [
        # One more contrast on a finished fit: small, repeated, latency.
        dict(name="contrast_20k_p4", call="test", G=20000, n=100000, p=4, patients=0, adjust="BH"),
        # A contrast on a clustered fit (max of the two p-values), wider design.
        dict(name="contrast_clustered_p12", call="test", G=20000, n=500000, p=12, patients=40, adjust="holm"),
        # The smallest fit: a marker panel with two covariates, host CSR.
        dict(name="fit_panel_p4", call="fit", design="continuous", G=200, n=2000, p=4, patients=0, od="MOM",
             counts="csr"),
        # A pilot experiment held as a dense double matrix, as R holds it.
        dict(name="fit_pilot_dense_p2", call="fit", design="pilot", G=2000, n=5000, p=2, patients=0, od="MLE",
             counts="dense"),
        # A sample with cell types and patients from the host (odd sizes).
        dict(name="fit_types_p12_host", call="fit", design="patients", G=3001, n=20011, p=12, patients=7, od="MLE",
             counts="csr"),
        # Continuous covariates at p = 4, counts resident on the GPU.
        dict(name="fit_cov_p4", call="fit_device", design="continuous", G=10000, n=100000, p=4, patients=0, od="MLE"),
        # Continuous covariates at p = 16 (batches, scores, ages), on the GPU.
        dict(name="fit_cov_p16", call="fit_device", design="continuous", G=8500, n=30000, p=16, patients=0, od="MLE"),
        # Bread and moment dispersion at given coefficients, wide covariates.
        dict(name="steps_cov_p24", call="steps", design="continuous", G=500, n=20000, p=24, patients=0),
        # Two conditions, a million cells, raw offsets (no size factors).
        dict(name="fit_binary_p2", call="fit_device", design="binary", G=4000, n=1000000, p=2, patients=0, od="MOM"),
        # Eleven cell types and forty patients: clustered sandwich.
        dict(name="fit_clustered_p12", call="fit_device", design="patients", G=4000, n=500000, p=12, patients=40,
             od="MOM"),
        # The atlas: 31 cell types, a million cells, dispersion by MLE.
        dict(name="fit_atlas_p32", call="fit_device", design="types", G=10000, n=1000000, p=32, patients=0, od="MLE"),
        # Several uneven problems (one per tissue) in one call, host CSR.
        dict(name="fit_batch_4", call="batch", design="types", G=1500, n=9000, p=8, patients=0, od="MLE", problems=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["test", "fit_small", "fit_host", "fit_host", "cov", "steps", "grouped", "grouped", "clustered"])
    od = rng.choice(["MOM", "MLE"])
    if kind == "test":
        return dict(call="test", G=_log_int(rng, 2000, 40000), n=_log_int(rng, 2000, 1000000), p=rng.randint(2, 32),
                    patients=rng.choice([0, 12]), adjust=rng.choice(["BH", "BY", "holm", "hochberg", "bonferroni"]))
    if kind == "fit_small":
        return dict(call="fit", design="continuous", G=rng.randint(60, 250), n=_log_int(rng, 400, 8000),
                    p=rng.randint(3, 8), patients=0, od=od, counts=rng.choice(["csr", "dense"]))
    if kind == "fit_host":
        design = rng.choice(["binary", "patients", "types"])
        return dict(call="fit", design=design, G=_log_int(rng, 300, 4000), n=_log_int(rng, 3000, 40000),
                    p=2 if design == "binary" else rng.randint(4, 14),
                    patients=rng.randint(3, 12) if design == "patients" else 0, od=od,
                    counts=rng.choice(["csr", "csr", "dense"]))
    if kind == "cov":
        p = rng.choice([4, 16])
        return dict(call="fit_device", design="continuous", p=p, patients=0, od=od,
                    G=rng.randint(9900, 10000) if p == 4 else rng.randint(8330, 8700),
                    n=_log_int(rng, 60000, 100000) if p == 4 else _log_int(rng, 12000, 30000))
    if kind == "steps":
        return dict(call="steps", design="continuous", G=_log_int(rng, 100, 1200), n=_log_int(rng, 3000, 30000),
                    p=rng.randint(9, 32), patients=0)
    if kind == "grouped":
        design = rng.choice(["binary", "types"])
        return dict(call="fit_device", design=design, G=_log_int(rng, 500, 6000), n=_log_int(rng, 60000, 1000000),
                    p=2 if design == "binary" else rng.randint(5, 32), patients=0, od=od)
    return dict(call="fit_device", design="patients", G=_log_int(rng, 500, 4000), n=_log_int(rng, 60000, 500000),
                p=rng.randint(4, 12), patients=rng.randint(5, 40), od=od)


# ----------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------
def _design(case, rng, n):
    p, cols = case["p"], [np.ones(n), (np.arange(n) % 2).astype(np.float64)]
    if case["design"] in ("types", "patients"):
        t = rng.integers(0, p - 1, n)
        cols += [(t == k).astype(np.float64) for k in range(1, p - 1)]
    else:
        cols += [rng.normal(0.0, 1.0, n) for _ in range(p - 2)]
    return np.stack(cols, 1)


def _model(case, seed, G, n):
    """Design, truth and cluster ends of one problem."""
    rng = np.random.default_rng([seed, G, n])
    X = _design(case, rng, n)
    p = X.shape[1]
    beta = np.zeros((G, p))
    loc, sd = _MEANS[case["design"]]
    types = p - 1 if case["design"] in ("types", "patients") else 1
    least = max(-5.3, math.log(40.0 * types / n))
    b0 = rng.normal(loc, sd, 64 * G)
    b0 = b0[(b0 > least) & (b0 < 5.0)][:G]
    beta[:, 0] = np.resize(b0, G) if len(b0) else least
    beta[0, 0] = 3.0
    beta[:, 1] = np.where(rng.random(G) < 0.1, rng.normal(0.0, 1.0, G), 0.0)
    beta[:, 2:] = rng.normal(0.0, 0.5 if case["design"] in ("types", "patients") else 0.2, (G, p - 2))
    theta = np.clip(rng.lognormal(0.0, 1.0, G), 0.05, 10.0)
    k, ends = case["patients"], None
    if k > 1:
        sizes = np.maximum(1, np.round(rng.dirichlet(np.full(k, 3.0)) * n).astype(np.int64))
        sizes[np.argmax(sizes)] += n - sizes.sum()
        ends = np.cumsum(sizes).astype(np.int32)
    return rng, X, beta, theta, ends


def _positive_counts(u, mu, th, gen):
    """Negative binomial counts given that they are positive: the inverse
    distribution function at u (above the mass of zero), entry by entry."""
    q = th * mu / (1 + th * mu)
    a = 1 / th
    pmf = torch.exp(-a * torch.log1p(th * mu))
    cdf = pmf.clone()
    y = torch.zeros_like(mu)
    at = torch.arange(mu.numel(), device=mu.device)
    for k in range(1, 33):
        pmf = pmf * q * (a + (k - 1)) / k
        cdf = cdf + pmf
        up = cdf < u
        y[at[~up]] = k
        at, u, pmf, cdf, q, a = at[up], u[up], pmf[up], cdf[up], q[up], a[up]
        if not at.numel():
            return y
    m, t = mu[at], th[at]
    big = torch.zeros_like(m)
    for _ in range(6):  # the tail: draws above 32
        big = torch.where(big > 32, big, torch.poisson(torch._standard_gamma(1 / t, generator=gen) * t * m, generator=gen))
    y[at] = big.clamp(33, 65535)
    return y


def _counts(seed, X, beta, theta, rng, ends):
    """CSR (gene-major) of one problem's counts on the GPU."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    n, G = X.shape[0], beta.shape[0]
    Xd, b = (torch.tensor(v, dtype=torch.float32, device=dev) for v in (X, beta))
    lsf = torch.tensor(rng.normal(0.0, 0.3, n), dtype=torch.float32, device=dev)
    th = torch.tensor(theta, dtype=torch.float32, device=dev)
    pat = pe = None
    if ends is not None:  # patients shift a gene's level
        pat = torch.tensor(np.repeat(np.arange(len(ends)), np.diff(ends, prepend=0)), device=dev)
        pe = torch.tensor(rng.normal(0.0, 0.3, (G, len(ends))), dtype=torch.float32, device=dev)
    rows, num, cols, vals = max(1, (1 << 27) // n), [], [], []
    for g in range(0, G, rows):
        eta = b[g:g + rows] @ Xd.T + lsf
        if pat is not None:
            eta += pe[g:g + rows][:, pat]
        mu, t = eta.exp_(), th[g:g + rows, None]
        u = torch.rand(mu.shape, device=dev, generator=gen)
        p0 = torch.exp(-torch.log1p(mu * t) / t)
        if g == 0:  # this gene is seen in every cell
            u[0] = torch.maximum(u[0], p0[0] + 1e-3)
        keep = u > p0
        num.append(keep.sum(1))
        at = keep.view(-1).nonzero().view(-1)
        r = torch.div(at, n, rounding_mode="floor")
        cols.append((at - r * n).to(torch.int32))
        y = _positive_counts(u.view(-1)[at], mu.view(-1)[at], th[g + r], gen)
        vals.append(y.to(torch.int32).to(torch.int16))  # the bits of uint16
        del eta, mu, u, p0, keep, at, r, y
    ptr = torch.zeros(G + 1, dtype=torch.int64, device=dev)
    ptr[1:] = torch.cumsum(torch.cat(num), 0)
    return ptr, torch.cat(cols), torch.cat(vals)


def _problem(case, seed, G=None, n=None):
    rng, X, beta, theta, ends = _model(case, seed, G or case["G"], n or case["n"])
    ptr, col, val = _counts(seed, X, beta, theta, rng, ends)
    return dict(X=X, beta=beta, theta=theta, ends=ends, ptr=ptr, col=col, val=val)


def _batch_sizes(case):
    return [(case["G"] + 700 * i, case["n"] // (1 << i) + 17 * i) for i in range(case["problems"])]


def _host_csr(d, n):
    return (d["ptr"].cpu().numpy(), d["col"].cpu().numpy(), d["val"].cpu().numpy().view(np.uint16), n)


def _dense64(d, n, rows=slice(None)):
    ptr = d["ptr"]
    g0, g1, _ = rows.indices(len(ptr) - 1)
    e0, e1 = int(ptr[g0]), int(ptr[g1])
    Y = torch.zeros((g1 - g0, n), dtype=torch.float64, device=ptr.device)
    r = torch.repeat_interleave(torch.arange(g1 - g0, device=ptr.device), ptr[g0 + 1:g1 + 1] - ptr[g0:g1])
    Y[r, d["col"][e0:e1].long()] = (d["val"][e0:e1].to(torch.int32) & 0xFFFF).double()
    return Y


def _labels(ends):
    return None if ends is None else np.repeat(np.arange(1, len(ends) + 1), np.diff(ends, prepend=0))


def _contrast(p):
    c = np.zeros(p)
    c[1] = 1.0
    return c


def prepare(case, seed):
    call, n, p = case["call"], case["n"], case["p"]
    if call == "test":
        rng = np.random.default_rng(seed)
        G = case["G"]
        A = rng.normal(0.0, 1.0, (G, p, p)) / math.sqrt(p)
        bread = (A @ A.transpose(0, 2, 1) + 0.3 * np.eye(p)) * rng.lognormal(0.0, 1.0, (G, 1, 1)) * (20.0 / n)
        beta = rng.normal(0.0, 1.0, (G, p)) * np.sqrt(np.einsum("gii->gi", bread)) * rng.choice(
            [0.7, 3.0], (G, 1), p=[0.8, 0.2])
        fit = dict(beta=beta, beta_sandwiches_null=bread, design_matrix=np.ones((n, p)),
                   beta_sandwiches=bread * rng.lognormal(0.3, 0.3, (G, 1, 1)) if case["patients"] else None)
        return dict(case=case, fit=fit, contrast=_contrast(p))
    if call == "batch":
        ds = [(_problem(case, seed * 64 + i, G, m), m) for i, (G, m) in enumerate(_batch_sizes(case))]
        return dict(case=case, problems=[(_host_csr(d, m), d["X"]) for d, m in ds])
    d = _problem(case, seed)
    if call == "fit":
        x = _dense64(d, n).cpu().numpy() if case["counts"] == "dense" else _host_csr(d, n)
        return dict(case=case, x=x, X=d["X"], clusters=_labels(d["ends"]))
    if call == "steps":
        return dict(case=case, x=_host_csr(d, n), X=d["X"], beta=d["beta"], theta=d["theta"], sf=_sf(case, seed))
    return _device_state(case, d)


def _sf(case, seed):
    return np.random.default_rng([seed, 7]).lognormal(0.0, 0.3, case["n"])


def _device_state(case, d):
    """A fit of counts that are on the GPU: the structures and result buffers
    that a program using the C ABI keeps."""
    G, n, p, dev = case["G"], case["n"], case["p"], torch.device("cuda")
    X = torch.tensor(np.ascontiguousarray(d["X"].T), device=dev)  # column-major
    counts = L.Counts()
    counts.format = L.COUNTS_CSR_U16
    counts.n_genes, counts.n_cells, counts.nnz = G, n, d["col"].numel()
    counts.values, counts.ptr, counts.idx = (d[k].data_ptr() for k in ("val", "ptr", "col"))
    opts = L.FitOpts()
    L.load().devil_fit_opts_default(C.byref(opts))
    opts.overdispersion = L.OD_MLE if case["od"] == "MLE" else L.OD_MOM
    opts.size_factors = L.SF_NONE if case["design"] == "binary" else L.SF_NORMED_SUM
    clustered = d["ends"] is not None
    f8, i4 = torch.float64, torch.int32
    shapes = dict(beta=((G, p), f8), theta=((G,), f8), iters=((G,), i4), bread=((G, p, p), f8), status=((G,), i4),
                  sf=((n,), f8), off=((n,), f8), pval=((G,), f8), adj=((G,), f8), lfc=((G,), f8))
    if clustered:
        shapes |= dict(sandwich=((G, p, p), f8), meat=((G, p, p), f8))
    out = {k: torch.zeros(s, dtype=t, device=dev) for k, (s, t) in shapes.items()}
    at = {k: C.c_void_p(v.data_ptr()) for k, v in out.items()}
    res = L.FitResult(at["beta"], at["theta"], at["iters"], None, at["bread"], at.get("sandwich"), None,
                      at["status"], at["sf"], at["off"], at.get("meat"))
    return dict(case=case, keep=(d["ptr"], d["col"], d["val"]), X=X, counts=counts, opts=opts, res=res, out=out, at=at,
                ends=d["ends"], contrast=_contrast(p), ctx=L.context())


# ----------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------
def _host_fit_outputs(f):
    return dict(beta=f["beta"], theta=f["overdispersion"], iters=f["iterations"]["beta_iters"],
                bread=f["beta_sandwiches_null"], status=f["status"], sf=f["size_factors"], off=f["offset_vector"],
                sandwich=f["beta_sandwiches"], meat=f["meat"])


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "test":
        r = dv.test_de(state["fit"], state["contrast"], pval_adjust_method=case["adjust"])
        return dict(pval=r["pval"], adj=r["adj_pval"], lfc=r["lfc"])
    if call == "batch":
        fits = dv.fit_devil_batch(state["problems"], overdispersion=case["od"], size_factors="normed_sum")
        return [_host_fit_outputs(f) for f in fits]
    if call == "fit":
        f = dv.fit_devil(state["x"], state["X"], clusters=state["clusters"], overdispersion=case["od"],
                         size_factors="normed_sum")
        return _host_fit_outputs(f)
    if call == "steps":
        bread = dv.compute_hessian(state["beta"], state["theta"], state["x"], state["X"], state["sf"])
        return dict(bread=bread, mom=dv.estimate_mom_dispersion(state["x"], state["X"], state["beta"], state["sf"]))
    lib, ctx, at, p = L.load(), state["ctx"], state["at"], case["p"]
    ends = state["ends"]
    ctx.check(lib.devil_fit_device(ctx.h, C.byref(state["counts"]), C.c_void_p(state["X"].data_ptr()), p,
                                   None if ends is None else ends.ctypes.data_as(C.c_void_p),
                                   0 if ends is None else len(ends), C.byref(state["opts"]), C.byref(state["res"])))
    ctx.check(lib.devil_test_de_device(ctx.h, case["G"], p, at["beta"], at["bread"], at.get("sandwich"), case["n"],
                                       state["contrast"].ctypes.data_as(C.c_void_p), L.ADJ_BH, 10.0, at["pval"],
                                       at["adj"], at["lfc"]))
    return state["out"]


def work(case):
    """What a pass cannot do without.  A fit reads its counts (6 bytes an
    entry; 8 bytes a value when dense) and design once and writes its results
    once; its operations are those of about a dozen Newton steps of X'WX per
    gene over the distinct (design row, size factor) terms it sums: the cells
    for continuous covariates, the nonzero counts otherwise."""
    call, G, n, p = case["call"], case["G"], case["n"], case["p"]
    mats = 2 if case["patients"] else 1
    if call == "test":
        return dict(bytes=8.0 * G * (p + mats * p * p + 3), flops=2.0 * G * mats * p * p)
    if call == "batch":
        sizes = _batch_sizes(case)
    else:
        sizes = [(G, n)]
    b = f = 0.0
    for g, m in sizes:
        loc, sd = _MEANS[case["design"]]
        dens = min(0.6, math.exp(loc + 0.25 * sd * sd))
        cov = case["design"] == "continuous"
        b += g * m * (8.0 if case.get("counts") == "dense" else 6.0 * dens) + 8.0 * m * p
        b += 8.0 * g * (p + 1 + mats * p * p)
        passes = 2 if call == "steps" else 12
        f += passes * (g * m * (p * (p + 1.0) + 2.0 * p) if cov else g * m * dens * 8.0)
    return dict(bytes=b, flops=f)


# ----------------------------------------------------------------------
# the same results in 64-bit arithmetic, with torch alone
# ----------------------------------------------------------------------
_MOST_CELLS = 1.1e9  # gene-cells that the 64-bit fit takes in reasonable time


def exact(case, seed):
    call = case["call"]
    if call == "test":
        return _exact_test(prepare(case, seed))
    if call == "batch":
        return [_exact_fit(_problem(case, seed * 64 + i, G, m), case, m) for i, (G, m) in enumerate(_batch_sizes(case))]
    if case["G"] * case["n"] > _MOST_CELLS or (case["design"] in ("types", "patients") and case["G"] * case["n"] > 2e8):
        return None
    d = _problem(case, seed)
    if call == "steps":
        t = _Fit(d, case["n"], sf=torch.tensor(_sf(case, seed), device="cuda"))
        beta, theta = (torch.tensor(d[k], device="cuda") for k in ("beta", "theta"))
        return dict(bread=t.bread(beta, theta)[0], mom=t.mom(beta))
    return _exact_fit(d, case, case["n"])


def _exact_fit(d, case, n):
    unit = case["call"] == "fit_device" and case["design"] == "binary"
    t = _Fit(d, n, sf=torch.ones(n, dtype=torch.float64, device="cuda") if unit else None)
    theta0 = t.theta0()
    beta, iters, status = t.irls(t.beta0(), theta0)
    mom = t.mom(beta)
    theta = mom if case["od"] == "MOM" else t.mle(beta)
    bread, scores = t.bread(beta, theta, d["ends"])
    sandwich = meat = None
    if d["ends"] is not None:
        k = len(d["ends"])
        meat = torch.einsum("gki,gkj->gij", scores, scores) * ((k / (k - 1.0) if k > 1 else 1.0) / n)
        sandwich = bread @ meat @ bread * n
    out = dict(beta=beta, theta=theta, iters=None, bread=bread, status=None, sf=t.sf, off=t.off, sandwich=sandwich,
               meat=meat)
    if case["call"] == "fit_device":
        r = _wald(beta, bread, sandwich, n, "BH")
        out |= dict(pval=r["pval"], adj=r["adj"], lfc=r["lfc"])
    return out


class _Fit:
    """The per-gene model of one problem, dense in FP64, a chunk of genes at a time."""

    def __init__(self, d, n, sf=None):
        self.d, self.n, self.G = d, n, len(d["ptr"]) - 1
        self.X = torch.tensor(d["X"], device="cuda")
        self.p = self.X.shape[1]
        i, j = torch.tril_indices(self.p, self.p, device="cuda")
        self.ij, self.Z = (i, j), self.X[:, i] * self.X[:, j]
        self.rows = max(1, int(2.5e8) // n)
        if sf is None:
            cs = torch.zeros(n, dtype=torch.float64, device="cuda")
            cs.index_add_(0, d["col"].long(), (d["val"].to(torch.int32) & 0xFFFF).double())
            sf = cs / torch.exp(torch.log(cs).mean())
        self.sf, self.off = sf, torch.log(sf)

    def chunks(self):
        for g in range(0, self.G, self.rows):
            s = slice(g, min(self.G, g + self.rows))
            yield s, _dense64(self.d, self.n, s)

    def mat(self, packed):
        M = torch.zeros(packed.shape[0], self.p, self.p, dtype=torch.float64, device="cuda")
        M[:, self.ij[0], self.ij[1]] = packed
        M[:, self.ij[1], self.ij[0]] = packed
        return M

    def mu(self, beta):
        return torch.exp(beta @ self.X.T + self.off)

    def theta0(self):
        out, moi = [], 1 / torch.exp(self.off).mean()
        for _, Y in self.chunks():
            m, v = Y.mean(1), Y.var(1)
            t = (v - moi * m) / (m * m)
            out.append(torch.where(torch.isnan(t) | (t < 0), torch.full_like(t, 0.01), t))
        return torch.cat(out)

    def beta0(self):
        inv = torch.linalg.inv(self.X.T @ self.X)
        return torch.cat([torch.log1p(Y / torch.exp(self.off)) @ self.X @ inv for _, Y in self.chunks()])

    def irls(self, beta, theta0, max_iter=200, tol=1e-3):
        beta, k_all, eps = beta.clone(), (1 / theta0.float().double()).float().double(), float(np.float32(tol))
        iters = torch.zeros(self.G, dtype=torch.int32, device="cuda")
        status = torch.ones_like(iters)
        for s, Y in self.chunks():
            act = torch.arange(s.start, s.stop, device="cuda")
            for it in range(1, max_iter + 1):
                k, w = k_all[act][:, None], 1 / self.mu(beta[act])
                w = (k + Y) / (1 + k * w) * w
                H, score = self.mat(w @ self.Z) * k[..., None], (w - 1) @ self.X * k
                step = torch.linalg.solve_ex(H, score)[0]
                beta[act] += step
                iters[act] = it
                nan, small = torch.isnan(step[:, 0]), torch.nan_to_num(step.abs()).amax(1) < eps
                status[act[nan]], status[act[small & ~nan]] = 2, 0
                on = ~(nan | small)
                if not bool(on.all()):
                    act, Y = act[on], Y[on]
                if not act.numel():
                    break
        return beta, iters, status

    def mom(self, beta):
        out = []
        for s, Y in self.chunks():
            mu = self.mu(beta[s])
            den = (mu * mu).sum(1)
            out.append(torch.clamp(self.n / (self.n - self.p) * ((Y - mu) ** 2 - mu).sum(1) / den, min=0.0))
        return torch.cat(out)

    def mle(self, beta):
        """The root of the Cox-Reid adjusted score in log theta, by bisection."""
        out, d = [], self.d
        for s, Y in self.chunks():
            mu, sum_y = self.mu(beta[s]), Y.sum(1)
            sp, mx = (Y * (Y - 1)).sum(1), Y.amax(1)
            e0, e1 = int(d["ptr"][s.start]), int(d["ptr"][s.stop])
            y = (d["val"][e0:e1].to(torch.int32) & 0xFFFF).double()
            r = torch.repeat_interleave(torch.arange(len(Y), device="cuda"),
                                        d["ptr"][s.start + 1:s.stop + 1] - d["ptr"][s.start:s.stop])
            eye = 1e-6 * torch.eye(self.p, dtype=torch.float64, device="cuda")

            def score(lt):
                th = torch.exp(lt)
                a = 1 / th
                x = mu * th[:, None]
                w = mu / (1 + x)
                ll = (torch.log1p(x) + (Y - mu) * th[:, None] / (1 + x)).sum(1)
                corr = torch.where(a > 1e5, sp / (2 * a), torch.zeros_like(a))
                ps = torch.zeros_like(a).index_add_(0, r, torch.digamma(y + a[r]) - torch.digamma(a)[r])
                dig = torch.where(mx * 1e6 < a, sum_y - corr, torch.minimum(ps * a, sum_y - corr))
                B, D = self.mat(w @ self.Z) + eye, self.mat(-(w * w) @ self.Z)
                cr = -0.5 * 0.99 * torch.linalg.solve_ex(B, D)[0].diagonal(dim1=1, dim2=2).sum(1)
                return a * ll - dig + cr * th

            lo = torch.full_like(sum_y, math.log(1e-8))
            hi = torch.full_like(sum_y, math.log(1e16))
            zero = (sum_y == 0) | (score(lo) < 0)
            for _ in range(52):
                mid = 0.5 * (lo + hi)
                up = score(mid) > 0
                lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
            out.append(torch.where(zero, torch.zeros_like(lo), torch.exp(0.5 * (lo + hi))))
        return torch.cat(out)

    def bread(self, beta, theta, ends=None):
        H, scores = [], []
        for s, Y in self.chunks():
            th, mu = theta[s][:, None], self.mu(beta[s])
            x = 1 + th * mu
            H.append(torch.linalg.inv_ex(self.mat((Y * th + 1) * mu / (x * x) @ self.Z))[0])
            if ends is not None:
                r, at = (Y - mu) / x, [0, *(int(e) for e in ends)]
                scores.append(torch.stack([r[:, a:b] @ self.X[a:b] for a, b in zip(at, at[1:])], 1))
        return torch.cat(H), torch.cat(scores) if scores else None


def _t_two_sided(t, df):
    """2 P(T > |t|) = I_{df/(df+t^2)}(df/2, 1/2), by Lentz's continued fraction."""
    t = np.abs(t)
    a0 = 0.5 * df
    x, omx = df / (df + t * t), t * t / (df + t * t)
    z = a0 + 0.5
    if a0 >= 100:  # log Gamma(a + 1/2) - log Gamma(a), Stirling's series term by term
        lg = (a0 - 0.5) * math.log1p(0.5 / a0) + 0.5 * math.log(z) - 0.5
        lg += (1 / z - 1 / a0) / 12 - (1 / z ** 3 - 1 / a0 ** 3) / 360 + (1 / z ** 5 - 1 / a0 ** 5) / 1260
    else:
        lg = math.lgamma(z) - math.lgamma(a0)
    lbeta = 0.5 * math.log(math.pi) - lg
    with np.errstate(all="ignore"):
        lx = np.where(x > 0.5, np.log1p(-omx), np.log(x))
        front = np.exp(a0 * lx + 0.5 * np.where(x > 0.5, np.log(omx), np.log1p(-x)) - lbeta)
        first = x < (a0 + 1) / (a0 + 2.5)

        def cf(a, b, v):
            c, d = np.ones_like(v), 1 / (1 - (a + b) * v / (a + 1))
            h = d.copy()
            for m in range(1, 4000):
                for e in (m * (b - m) * v / ((a + 2 * m - 1) * (a + 2 * m)),
                          -(a + m) * (a + b + m) * v / ((a + 2 * m) * (a + 2 * m + 1))):
                    d, c = 1 / (1 + e * d), 1 + e / c
                    h *= d * c
                if np.all(np.abs(d * c - 1) < 1e-16):
                    break
            return h

        p = np.where(first, front * cf(a0, 0.5, np.where(first, x, 0.1)) / a0,
                     1 - front * cf(0.5, a0, np.where(first, 0.1, omx)) / 0.5)
    return np.where(t == 0, 1.0, p)


def _wald(beta, bread, sandwich, n, adjust):
    b, H = (np.asarray(v.cpu() if torch.is_tensor(v) else v) for v in (beta, bread))
    c = _contrast(b.shape[1])
    l = b @ c
    var = [np.einsum("i,gij,j->g", c, H, c)]
    if sandwich is not None:
        var.append(np.einsum("i,gij,j->g", c, np.asarray(sandwich.cpu() if torch.is_tensor(sandwich) else sandwich), c))
    with np.errstate(all="ignore"):
        p = np.max([_t_two_sided(l / np.sqrt(v), n - 2.0) for v in var], 0)
    return dict(pval=p, adj=_adjust(p, adjust), lfc=np.clip(l / math.log(2.0), -10.0, 10.0))


def _adjust(p, how):
    out, ok = p.copy(), ~np.isnan(p)
    v = p[ok]
    m, o = len(v), np.argsort(v, kind="stable")
    s, i = v[o], np.arange(1, len(v) + 1.0)
    if how == "bonferroni":
        q = m * s
    elif how == "holm":
        q = np.maximum.accumulate((m + 1 - i) * s)
    else:
        f = {"BH": m / i, "BY": m / i * np.sum(1 / i), "hochberg": m + 1 - i}[how]
        q = np.minimum.accumulate((f * s)[::-1])[::-1]
    back = np.empty(m)
    back[o] = np.minimum(1.0, q)
    out[ok] = back
    return out


def _exact_test(state):
    f, case = state["fit"], state["case"]
    return _wald(f["beta"], f["beta_sandwiches_null"], f["beta_sandwiches"], case["n"], case["adjust"])
