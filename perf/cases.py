"""The work this engine is timed on: the calls a genome-wide association user makes, over the range they make them in.

A case names one entry point (`kind`), the problem (n individuals, t traits, wXL covariates, wXR columns per SNP) and
the SNPs of one pass (x for a block already on the device, m for a job from host memory).  Inputs follow the
distributions of fgls_gb300/datagen.py: genotypes Binomial(2, f) with f ~ U(0.05, 0.5), kinship G G^T / 5000 + 1e-3 I
of standardised genotypes, an intercept and normal covariates, h ~ U(0.1, 0.9), sigma ~ U(0.5, 2), and traits with
covariance sigma (h Phi + (1 - h) I).  Dosages (imputed genotypes, real values in [0, 2]) go to the FP64 path only:
the split path is defined for hard calls.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cugwas-proto_gb300"))
from fgls_gb300 import Batch, Engine  # noqa: E402

MARKERS = 5000  # kinship markers, as in fgls_gb300/datagen.py
F64 = torch.float64


def listed():
    return [
        # The multi-trait scan that the benchmark measures: one resident block of n = 10k, 100 traits, split precision.
        dict(name="eigen_split_10k_t100", kind="eigen", precision="split", geno="f64", n=10000, t=100, wXL=3, wXR=1,
             x=16384),
        # A small study with one trait and a short block of byte genotypes: launches and latency.
        dict(name="eigen_split_small", kind="eigen", precision="split", geno="u8", n=750, t=1, wXL=3, wXR=1, x=512),
        # The default precision of the engine and of the drop-in on a mid-size study with a few traits.
        dict(name="eigen_fp64_5k_t16", kind="eigen", precision="fp64", geno="f64", n=5000, t=16, wXL=3, wXR=1, x=4096),
        # The reference's own GPU workload: one trait, n = 10k, streamed 4096-SNP blocks, FP64; imputed dosages.
        dict(name="chol_fp64_10k_dosage", kind="chol", precision="fp64", geno="dosage", n=10000, t=1, wXL=3, wXR=1,
             x=4096),
        # The same workload on the split path with packed hard calls.
        dict(name="chol_split_10k_packed", kind="chol", precision="split", geno="packed", n=10000, t=1, wXL=3, wXR=1,
             x=4096),
        # A tiny interactive query through host memory: two columns per SNP, an odd block, FP64.
        dict(name="chol_fp64_tiny_host", kind="chol_host", precision="fp64", geno="f64", n=301, t=1, wXL=3, wXR=2, x=37),
        # The backward direction: gradients of the effects by h, sigma and the traits.
        dict(name="adjoint_5k_t16", kind="adjoint", precision="fp64", geno="f64", n=5000, t=16, wXL=3, wXR=1, x=4096),
        # Meta-analysis: many cohorts of uneven size advanced together.
        dict(name="cohorts_16", kind="cohorts", precision="split", geno="u8", count=16, n_lo=500, n_hi=4000, t=2,
             x=2048),
        # Variance components of many traits before the scan.
        dict(name="reml_fit_4k_t100", kind="reml", precision="fp64", geno="f64", n=4001, t=100, wXL=4, wXR=1, x=64),
        # A whole small study from host memory: eigendecomposition, null models, scan with SE and p-values; FP64.
        dict(name="job_eigen_fp64_2k", kind="job_eigen", precision="fp64", geno="f64", n=2003, t=5, wXL=4, wXR=1,
             m=5001),
        # A whole multi-trait study from a packed genotype file's contents, split precision.
        dict(name="job_eigen_split_5k", kind="job_eigen", precision="split", geno="packed", n=5000, t=32, wXL=3, wXR=1,
             m=20000),
        # A whole single-trait study: factorization of the trait's covariance and the scan, split precision.
        dict(name="job_chol_split_6k", kind="job_chol", precision="split", geno="u8", n=6000, t=1, wXL=2, wXR=1,
             m=12000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eigen", "eigen", "chol", "chol", "chol_host", "adjoint", "cohorts", "reml", "job_eigen",
                       "job_chol"])
    precision = rng.choice(["split", "fp64"])
    geno = rng.choice(["f64", "u8", "packed"] if precision == "split" else ["f64", "u8", "packed", "dosage"])
    c = dict(kind=kind, precision=precision, geno=geno, n=_log_int(rng, 300, 6000), t=_log_int(rng, 1, 120),
             wXL=rng.randint(1, 6), wXR=rng.choice([1, 1, 1, 2]) if precision == "fp64" else 1)  # split: one column
    if kind == "cohorts":
        return dict(kind=kind, precision="split", geno=rng.choice(["u8", "f64"]), count=rng.randint(3, 16),
                    n_lo=_log_int(rng, 200, 800), n_hi=_log_int(rng, 900, 4000), t=rng.randint(1, 2),
                    x=_log_int(rng, 200, 2048))
    if kind in ("chol", "job_chol", "chol_host"):
        c["t"] = 1
    if kind == "chol":
        c["n"] = _log_int(rng, 300, 10000)
    if kind in ("adjoint", "reml"):
        c.update(precision="fp64", geno="f64", wXR=1)
    if kind == "adjoint":
        c["t"] = _log_int(rng, 1, 16)
    if kind == "chol_host":
        c.update(geno="f64", n=_log_int(rng, 200, 2000), x=_log_int(rng, 16, 512))
    elif kind == "reml":
        c["x"] = 64
    elif kind in ("job_eigen", "job_chol"):
        c.update(geno=rng.choice(["u8", "packed"]) if precision == "split" else "f64",
                 m=_log_int(rng, 500, 12000), t=min(c["t"], 40), n=min(c["n"], 4500))
    else:
        # one pass of the FP64 path stays below the largest listed one
        c["x"] = _log_int(rng, 100, 4096) if precision == "fp64" else _log_int(rng, 100, 16384)
    return c


def _problem(case, seed):
    """(generator, Phi n x n symmetric, XL wXL x n, Y t x n, h, sigma) on the GPU."""
    n, t, wXL = case["n"], case["t"], case["wXL"]
    g = torch.Generator("cuda").manual_seed(seed)
    kw = dict(generator=g, device="cuda", dtype=F64)
    f = 0.05 + 0.45 * torch.rand(MARKERS, **kw).float()
    u = lambda: torch.rand(n, MARKERS, generator=g, device="cuda")  # noqa: E731
    G = ((u() < f).to(torch.uint8) + (u() < f).to(torch.uint8)).to(F64)
    sd = G.std(dim=0, unbiased=False)
    G = (G - G.mean(dim=0)) / torch.where(sd > 0, sd, torch.ones_like(sd))
    Phi = (G @ G.T).div_(MARKERS)
    Phi = torch.tril(Phi) + torch.tril(Phi, -1).T
    Phi.diagonal().add_(1e-3)
    h = 0.1 + 0.8 * torch.rand(t, **kw)
    sigma = 0.5 + 1.5 * torch.rand(t, **kw)
    Y = (G @ torch.randn(MARKERS, t, **kw)).mul_((h * sigma / MARKERS).sqrt())
    Y += torch.randn(n, t, **kw) * (h * sigma * 1e-3 + (1 - h) * sigma).sqrt()
    XL = torch.randn(wXL, n, **kw)
    XL[0] = 1.0
    return g, Phi, XL, Y.T.contiguous(), h, sigma


def _hard_calls(g, n, cols):
    f = 0.05 + 0.45 * torch.rand(cols, 1, generator=g, device="cuda")
    out = torch.empty(cols, n, dtype=torch.uint8, device="cuda")
    for a in range(0, cols, 4096):
        k = out[a:a + 4096]
        u = lambda: torch.rand(k.shape, generator=g, device="cuda") < f[a:a + 4096]  # noqa: E731
        k.copy_(u().to(torch.uint8) + u().to(torch.uint8))
    return out


def _genotypes(g, case, n, cols):
    """(as the call takes them, the values as FP64-convertible columns x n)."""
    calls = _hard_calls(g, n, cols)
    if case["geno"] == "u8":
        return calls, calls
    if case["geno"] == "f64":
        return calls.to(F64), calls
    if case["geno"] == "dosage":
        d = (calls.to(F64) + 0.2 * torch.randn(cols, n, generator=g, device="cuda", dtype=F64)).clamp_(0.0, 2.0)
        return d, d
    code = torch.tensor([3, 2, 0], dtype=torch.uint8, device="cuda")  # 2-bit .bed codes of 0, 1, 2 copies
    quads = torch.zeros(cols, -(-n // 4) * 4, dtype=torch.uint8, device="cuda")
    for a in range(0, cols, 4096):
        quads[a:a + 4096, :n] = code[calls[a:a + 4096].long()]
    q = quads.view(cols, -1, 4)
    return q[..., 0] | (q[..., 1] << 2) | (q[..., 2] << 4) | (q[..., 3] << 6), calls


def _host(x):
    """A host array in the orientation the engine takes: x (k x n) -> n x k, column-major."""
    return x.cpu().numpy().T


def _pinned(x):
    return torch.empty(x.shape, dtype=x.dtype, pin_memory=True).copy_(x)


def _cohorts(case):
    """(n, wXL) of each cohort: sizes spread over the logarithm, every 3..8 predictors."""
    k = case["count"]
    lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
    return [(int(math.exp(lo + (hi - lo) * i / max(1, k - 1))), 2 + (5 * i + i // 6) % 6) for i in range(k)]


def _cohort_parts(case, seed):
    for i, (n, wXL) in enumerate(_cohorts(case)):
        c = dict(case, n=n, wXL=wXL, wXR=1)
        g, *rest = _problem(c, seed * 1009 + i)
        yield c, rest, _genotypes(g, c, n, case["x"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "cohorts":
        parts, descs = [], []
        for c, (Phi, XL, Y, h, sigma), (geno, _) in _cohort_parts(case, seed):
            descs.append(dict(Phi=_host(Phi), XL=_host(XL), Y=_host(Y), h=h.cpu().numpy(), sigma=sigma.cpu().numpy()))
            p = c["wXL"] + 1
            parts.append((geno, torch.empty(c["t"], case["x"], p, dtype=F64, device="cuda"),
                          torch.empty(c["t"], case["x"], p, p, dtype=F64, device="cuda")))
        batch = Batch(descs, x_b=case["x"], genotypes_u8=case["geno"] == "u8")
        ptr = [[a.data_ptr() for a in part] for part in zip(*parts)]
        return dict(kind=kind, batch=batch, parts=parts, ptr=ptr, xs=[case["x"]] * len(parts))
    n, t, wXR, p = case["n"], case["t"], case["wXR"], case["wXL"] + case["wXR"]
    g, Phi, XL, Y, h, sigma = _problem(case, seed)
    job = kind in ("job_eigen", "job_chol")
    m = case["m"] if job else case["x"]
    eigen = kind not in ("chol", "chol_host", "job_chol")
    problem = [_host(Phi), _host(XL), _host(Y), h.cpu().numpy(), sigma.cpu().numpy()]
    del Phi
    e = Engine(n, case["wXL"], wXR, t, min(m, 4096) if job else m, "eigen" if eigen else "chol", case["precision"])
    s = dict(kind=kind, engine=e, problem=problem, m=m, geno=case["geno"])
    if kind != "reml":
        geno, _ = _genotypes(g, case, n, m * wXR)
        s["x"] = _host(geno) if kind == "chol_host" or job and case["geno"] == "f64" else _pinned(geno) if job else geno
        del geno
    if job:
        s["out"] = (torch.empty(t, m, p, dtype=F64, pin_memory=True), torch.empty(t, m, p, p, dtype=F64, pin_memory=True))
        return s
    e.set_problem(*problem)
    s["problem"] = None
    if not eigen:
        e.select_trait(0)
    if kind == "adjoint":
        s["bbar"] = torch.randn(t, m, p, generator=g, device="cuda", dtype=F64)
    elif kind in ("eigen", "chol"):
        s["out"] = (torch.empty(t, m, p, dtype=F64, device="cuda"), torch.empty(t, m, p, p, dtype=F64, device="cuda"))
        s["strides"] = (m * p, m * p * p)
    return s


def run(s):
    kind = s["kind"]
    if kind == "cohorts":
        s["batch"].step(s["ptr"][0], s["xs"], s["ptr"][1], s["ptr"][2])
        return [part[1:] for part in s["parts"]]
    e = s["engine"]
    if kind in ("eigen", "chol"):
        B, V = s["out"]
        e.run_block_device(s["x"].data_ptr(), s["m"], B.data_ptr(), V.data_ptr(), *s["strides"],
                           u8=s["geno"] == "u8", packed=s["geno"] == "packed")
        return s["out"]
    if kind == "chol_host":
        B, V = e.run_block(s["x"])
        return B, V
    if kind == "adjoint":
        bbar = s["bbar"]
        e.adjoint_reset()
        e.adjoint_block_device(s["x"].data_ptr(), s["m"], bbar.data_ptr(), bbar.stride(0))
        dh, dsigma, dY = e.adjoint_read()
        # one output: the effects do not depend on sigma, so its gradient alone is nothing but rounding
        return torch.stack([torch.from_numpy(dh), torch.from_numpy(dsigma)]), dY
    if kind == "reml":
        h, sigma, ll, dll = e.reml_fit()
        # the gradient is nothing but rounding at an inner maximum: it goes with the value
        return h, sigma, torch.stack([torch.from_numpy(ll), torch.from_numpy(dll)])
    e.set_problem(*s["problem"])
    if kind == "job_chol":
        e.select_trait(0)
    if s["geno"] == "f64":
        return e.run_snps_compact(s["x"])
    B, V = s["out"]
    e.run_snps_genotypes_ptr(s["x"].data_ptr(), s["m"], B.data_ptr(), V.data_ptr(), packed=s["geno"] == "packed")
    return s["out"]


def work(case):
    """Bytes: genotypes and the factor read once, effects and covariances written once.  Operations: the whitening of
    the genotypes, the Gram terms, and for jobs the factorization (4/3 n^3 and 2 n^3 of an eigendecomposition with
    vectors, n^3 / 3 of a Cholesky factorization)."""
    if case["kind"] == "cohorts":
        parts = [work(dict(kind="chol", geno=case["geno"], n=n, t=1, wXL=w, wXR=1, x=case["x"])) for n, w in _cohorts(case)]
        g = {"u8": 1, "f64": 8}[case["geno"]]
        again = sum(n * case["x"] * g for n, _ in _cohorts(case)) * (case["t"] - 1)  # one read serves all traits
        return {"bytes": case["t"] * sum(w["bytes"] for w in parts) - again,
                "flops": case["t"] * sum(w["flops"] for w in parts)}
    n, t, wXL, wXR, kind = case["n"], case["t"], case["wXL"], case["wXR"], case["kind"]
    p = wXL + wXR
    if kind == "reml":
        return {"bytes": 8.0 * n * (t + wXL + 1), "flops": 64.0 * t * n * (wXL + 2) * (wXL + 3)}
    m = case.get("m", case.get("x"))
    cols = m * wXR
    eigen = kind in ("eigen", "adjoint", "job_eigen")
    size = {"f64": 8.0, "dosage": 8.0, "u8": 1.0, "packed": 0.25}[case["geno"]]
    gram = 2.0 * n * cols * t * (1 + wXL + wXR)
    factor = 8.0 * n * n * (1.0 if eigen else 0.5)
    flops = (2.0 if eigen else 1.0) * n * n * cols + gram
    if kind == "adjoint":  # three weighted Gram blocks, the effects' cotangent in, the gradient by the traits out
        return {"bytes": size * n * cols + 2 * factor + 8.0 * t * m * p + 16.0 * n * t,
                "flops": flops + 2 * gram + 2.0 * n * t * m + 2.0 * n * n * t}
    out = 8.0 * t * m * (3 * p if kind == "job_eigen" and case["geno"] == "f64" else p + p * p)
    if kind.startswith("job"):
        flops += (10.0 / 3.0 if eigen else 1.0 / 3.0) * n ** 3
    return {"bytes": size * n * cols + factor + out, "flops": flops}


def _gls(Phi, XL, Y, h, sigma, X, wXR):
    """B (t, m, p) and V (t, m, p, p: lower triangle stored by columns, SE on the diagonal) in FP64."""
    n, wXL, t = Phi.shape[0], XL.shape[0], Y.shape[0]
    m = X.shape[0] // wXR
    p = wXL + wXR
    B = torch.empty(t, m, p, dtype=F64)
    V = torch.empty(t, m, p, p, dtype=F64)
    eig = torch.linalg.eigh(Phi) if t > 4 else None
    for j in range(t):
        if eig is None:
            M = Phi * (h[j] * sigma[j])
            M.diagonal().add_((1 - h[j]) * sigma[j])
            L = torch.linalg.cholesky(M)
            del M
            turn = lambda a: torch.linalg.solve_triangular(L, a.T, upper=False)  # noqa: E731
            weight = torch.ones(n, 1, device="cuda", dtype=F64)
        elif j == 0:
            turn = lambda a: eig[1].T @ a.T  # noqa: E731
        if eig is not None:
            weight = (1.0 / (sigma[j] * (h[j] * eig[0] + 1 - h[j])))[:, None]
            if j == 0:
                rotated = torch.cat([turn(X[a:a + 2048].to(F64)) for a in range(0, m * wXR, 2048)], dim=1)
                tl_all, ty_all = turn(XL), turn(Y)
            tl, ty = tl_all, ty_all[:, j:j + 1]
        else:
            tl, ty = turn(XL), turn(Y[j:j + 1])
        null = torch.linalg.solve(tl.T @ (weight * tl), tl.T @ (weight * ty))
        res = ty - tl @ null
        var = (weight * res * res).sum() / (n - wXL)
        for a in range(0, m, 2048):
            k = min(2048, m - a)
            if eig is None:
                xr = turn(X[a * wXR:(a + k) * wXR].to(F64))
            else:
                xr = rotated[:, a * wXR:(a + k) * wXR]
            wx = weight * xr
            S = torch.empty(k, p, p, device="cuda", dtype=F64)
            S[:, :wXL, :wXL] = tl.T @ (weight * tl)
            lr = (tl.T @ wx).T.reshape(k, wXR, wXL)
            S[:, wXL:, :wXL], S[:, :wXL, wXL:] = lr, lr.transpose(1, 2)
            x3, w3 = xr.reshape(n, k, wXR), wx.reshape(n, k, wXR)
            for c in range(wXR):
                for d in range(wXR):
                    S[:, wXL + c, wXL + d] = (x3[:, :, c] * w3[:, :, d]).sum(0)
            rhs = torch.empty(k, p, 1, device="cuda", dtype=F64)
            rhs[:, :wXL, 0] = (tl.T @ (weight * ty))[:, 0]
            rhs[:, wXL:, 0] = (ty.T @ wx).reshape(k, wXR)
            inv = torch.linalg.inv(S) * var
            B[j, a:a + k] = torch.linalg.solve(S, rhs)[:, :, 0].cpu()
            v = torch.tril(inv)
            v.diagonal(dim1=1, dim2=2).sqrt_()
            V[j, a:a + k] = v.transpose(1, 2).cpu()
    return B, V


def _exact_adjoint(case, seed):
    g, Phi, XL, Y, h, sigma = _problem(case, seed)
    n, t, wXL, x = case["n"], case["t"], case["wXL"], case["x"]
    X = _genotypes(g, case, n, x)[1].to(F64)
    bbar = torch.randn(t, x, wXL + 1, generator=g, device="cuda", dtype=F64)
    w, Z = torch.linalg.eigh(Phi)
    R, tl = Z.T @ X.T, Z.T @ XL.T
    RR = R * R
    grads = []
    for j in range(t):
        hj, sj, yj = (a.clone().requires_grad_() for a in (h[j], sigma[j], Y[j]))
        d = 1.0 / (sj * (hj * w + 1 - hj))
        ty = Z.T @ yj
        S = torch.zeros(x, wXL + 1, wXL + 1, device="cuda", dtype=F64)
        lr = R.T @ (d[:, None] * tl)
        top = torch.cat([(tl.T @ (d[:, None] * tl)).expand(x, wXL, wXL), lr[:, :, None]], dim=2)
        low = torch.cat([lr[:, None, :], (RR.T @ d)[:, None, None]], dim=2)
        S = torch.cat([top, low], dim=1)
        rhs = torch.cat([(tl.T @ (d * ty)).expand(x, wXL), (R.T @ (d * ty))[:, None]], dim=1)
        beta = torch.linalg.solve(S, rhs[:, :, None])[:, :, 0]
        grads.append(torch.autograd.grad((beta * bbar[j]).sum(), (hj, sj, yj)))
    return torch.stack([torch.stack([a[0] for a in grads]), torch.stack([a[1] for a in grads])]), \
        torch.stack([a[2] for a in grads], dim=1)


def _exact_reml(case, seed):
    """The best of the profiled likelihood's maxima on a 64-point grid of h, its brackets bisected on the gradient."""
    _, Phi, XL, Y, _, _ = _problem(case, seed)
    n, t, wXL = case["n"], case["t"], case["wXL"]
    w, Z = torch.linalg.eigh(Phi)
    x, y = Z.T @ XL.T, Z.T @ Y.T

    def at(h):  # h (t): likelihood, gradient and sigma of every trait
        den = 1 + h[None, :] * (w - 1)[:, None]
        d = 1 / den
        c = -(w - 1)[:, None] * d * d
        G = torch.einsum("la,lt,lb->tab", x, d, x)
        b = torch.linalg.solve(G, torch.einsum("la,lt->ta", x, d * y)[:, :, None])[:, :, 0]
        r = y - x @ b.T
        q = (d * r * r).sum(0)
        trace = torch.linalg.solve(G, torch.einsum("la,lt,lb->tab", x, c, x)).diagonal(dim1=1, dim2=2).sum(1)
        s = q / (n - wXL)
        ll = -0.5 * ((n - wXL) * s.log() + den.log().sum(0) + torch.logdet(G) + (n - wXL))
        return ll, -0.5 * ((n - wXL) * (c * r * r).sum(0) / q - (c / d).sum(0) + trace), s

    grid = torch.linspace(0.0, 1.0 - 1e-5, 64, dtype=F64, device="cuda")
    values = [at(h.expand(t)) for h in grid]
    ll, dll = torch.stack([v[0] for v in values]), torch.stack([v[1] for v in values])
    rising = (dll[:-1] > 0) & (dll[1:] <= 0)
    score = torch.where(rising, torch.maximum(ll[:-1], ll[1:]), torch.full_like(ll[1:], -math.inf))
    k = score.argmax(0)
    lo, hi = grid[k], grid[k + 1]
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        up = at(mid)[1] > 0
        lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
    h = 0.5 * (lo + hi)
    ends = torch.stack([torch.where(dll[0] <= 0, ll[0], -math.inf * torch.ones_like(ll[0])),
                        torch.where(dll[-1] >= 0, ll[-1], -math.inf * torch.ones_like(ll[0]))])
    inner = torch.where(rising.any(0), at(h)[0], -math.inf * torch.ones_like(ll[0]))
    h = torch.where(ends.amax(0) > inner, torch.where(ends[0] >= ends[1], grid[0], grid[-1]), h)
    ll, dll, s = at(h)
    return h, s, torch.stack([ll, dll])


def exact(case, seed):
    kind = case["kind"]
    if kind == "cohorts":
        return [_gls(Phi, XL, Y, h, sigma, X, 1) for _, (Phi, XL, Y, h, sigma), (_, X) in _cohort_parts(case, seed)]
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind == "reml":
        return _exact_reml(case, seed)
    g, Phi, XL, Y, h, sigma = _problem(case, seed)
    m = case.get("m", case.get("x"))
    X = _genotypes(g, case, case["n"], m * case["wXR"])[1]
    B, V = _gls(Phi, XL, Y, h, sigma, X, case["wXR"])
    if kind == "chol_host":
        return B, V.transpose(2, 3)
    if kind == "job_eigen" and case["geno"] == "f64":
        SE = V.diagonal(dim1=2, dim2=3).contiguous()
        return B, SE, torch.erfc((B / SE).abs() / math.sqrt(2.0))
    return B, V
