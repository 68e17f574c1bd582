"""Performance cases: the calls a user of this framework makes, over the sizes it is used at.

The framework fits SAIGE's null model.  A program loads a PLINK cohort (``setgeno``), selects an
engine for the GRM products (a resident GRM from ``grm_build``, or the subset-exact engine, which
applies each phenotype's own GRM through the genotype matrix), and then either drives the fit
itself through the drop-ins of the reference's Rcpp entry points (``getCoefficients``,
``GetTrace_q``, ``getAIScore`` ..., FP32 vectors at the boundary as in the reference) or hands whole
phenotypes to the batched driver (``native.fit_batch``).  Cohorts run from the reference's 1,000-sample
example to biobank size (100,000 samples by 150,000 markers); 1-2% of the calls are missing.

``exact`` restates each call in FP64 with plain torch: the operator Z Z' / M is applied from the
2-bit genotypes, and the solves stop by the same rule (sum r^2 <= tol).
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "saige-gpu_gb300"))

from saigegpu import (Context, GRM_BF16X3_TC, GRM_FP32_SIMT, MV_BF16X3_TC, MV_SUBSET_EXACT,  # noqa: E402
                      native, prep, serve)

TOL_PCG, MAXITER_PCG, NRUN, CUTOFF, PROBE_SEED = 1e-5, 500, 30, 0.0025, 200


def listed():
    return [
        # K b on the reference's example cohort size, every default: the smallest call there is
        {"name": "product_example", "call": "product", "engine": "default", "n": 1000, "m": 10000, "miss": 0.01},
        # one Sigma^-1 b on a resident split-BF16 GRM (getPCG1ofSigmaAndVector, as the R driver calls it)
        {"name": "solve_cohort_20k", "call": "solve", "engine": "bf16x3", "n": 20000, "m": 30000, "miss": 0.02},
        # getCoefficients on a ragged mid-size cohort in the subset-exact engine: four right-hand sides
        {"name": "coef_odd_20k", "call": "coef", "engine": "subset", "n": 20011, "m": 30007, "miss": 0.02},
        # coefficients with two of the 22 chromosomes left out in turn, as LOCO runs them after a fit
        {"name": "loco_50k", "call": "loco", "engine": "subset", "n": 50000, "m": 100000, "miss": 0.01},
        # the Hutchinson trace of one quantitative AI-REML iteration: 30 probes, solved and multiplied
        {"name": "trace_50k", "call": "trace", "engine": "subset", "n": 50000, "m": 100000, "miss": 0.01},
        # the AI score of one binary AI-REML iteration at biobank size: the largest single call
        {"name": "ai_100k", "call": "ai", "engine": "subset", "n": 100000, "m": 150000, "miss": 0.02},
        # the AI score of a quantitative iteration on a resident split-BF16 GRM
        {"name": "ai_cohort_24k", "call": "ai_q", "engine": "bf16x3", "n": 24576, "m": 30000, "miss": 0.02},
        # loading a cohort from a .bed image in host memory: decode, QC, re-pack, diagonal
        {"name": "setgeno_20k", "call": "setgeno", "engine": "none", "n": 20011, "m": 30007, "miss": 0.02},
        # the default GRM build of a small cohort, read back
        {"name": "grm_default_2k", "call": "grm", "engine": "none", "n": 2000, "m": 5000, "miss": 0.01},
        # the split-BF16 GRM build of a mid-size cohort and its first product
        {"name": "grm_split_20k", "call": "build", "engine": "none", "n": 20000, "m": 30000, "miss": 0.02},
        # eight masked phenotypes fit in one batch on a small cohort, where latency and launches count
        {"name": "fits_2k", "call": "fits", "engine": "subset", "n": 2000, "m": 5000, "miss": 0.01, "phenos": 8},
        # a batch of masked phenotypes on the plain method's cohort size: the batched driver's main use
        {"name": "fits_50k", "call": "fits", "engine": "subset", "n": 50000, "m": 100000, "miss": 0.01, "phenos": 16},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    call = rng.choice(["product", "solve", "coef", "coef", "loco", "trace", "ai", "ai_q", "setgeno", "grm", "build",
                       "fits"])
    engine = {"setgeno": "none", "grm": "none", "build": "none", "coef": "subset", "loco": "subset",
              "fits": "subset"}.get(call)
    if engine is None:
        engine = rng.choice(["subset", "subset", "bf16x3", "default"])
    case = {"call": call, "engine": engine, "miss": rng.choice([0.0, 0.01, 0.02])}
    if call == "grm":
        case.update(n=_log(rng, 500, 4000), m=_log(rng, 2000, 12000))
    elif call == "fits":
        case.update(n=_log(rng, 1000, 50000), m=_log(rng, 5000, 100000), phenos=rng.randint(2, 16))
    elif engine == "default":
        case.update(n=_log(rng, 500, 6000), m=_log(rng, 2000, 15000))
    elif engine in ("bf16x3", "none"):
        case.update(n=_log(rng, 1000, 24576), m=_log(rng, 5000, 45000))
    else:
        case.update(n=_log(rng, 1000, 100000), m=_log(rng, 5000, 150000))
    return case


# ------------------------------------------------------------------------------------ inputs
def _gen(seed, stream):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 64 + stream)


def _bed(n, m, miss, seed, rare=False):
    """A .bed image on the GPU: p ~ U(0.01, 0.5), Hardy-Weinberg genotypes, calls missing at random."""
    nb = (n + 3) // 4
    g = _gen(seed, 0)
    img = torch.empty(3 + nb * m, dtype=torch.uint8, device="cuda")
    img[:3] = torch.tensor([0x6C, 0x1B, 0x01], dtype=torch.uint8)
    body = img[3:].view(m, nb)
    p = 0.01 + 0.49 * torch.rand(m, 1, generator=g, device="cuda")
    if rare:  # every 20th marker far below the frequency threshold, none near it: as many pass for any seed
        p = p * 0.9 + 0.05
        p[::20] = 0.001
    t1 = miss + (1 - miss) * (1 - p) ** 2
    t2 = miss + (1 - miss) * (1 - p * p)
    w = torch.tensor([1, 4, 16, 64], dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 28) // (4 * nb))
    for i in range(0, m, step):
        k = min(step, m - i)
        u = torch.rand(k, 4 * nb, generator=g, device="cuda")
        a, b = u >= t1[i:i + k], u >= t2[i:i + k]
        # packed fields: missing 1, no copy 3, one copy 2, two copies 0
        f = torch.where(b, 0, torch.where(a, 2, 3)).to(torch.uint8)
        if miss:
            f.masked_fill_(u < miss, 1)
        if n % 4:
            f[:, n:] = 0
        body[i:i + k] = (f.view(k, nb, 4) * w).sum(2, dtype=torch.uint8)
    return img


def _normal(n, seed, stream, cols=1):
    x = torch.randn(cols, n, generator=_gen(seed, stream), device="cuda", dtype=torch.float64)
    return x.T.cpu().numpy()


def _genetic(img, n, m, seed, k):
    """k standardised polygenic values from 1,000 of the markers."""
    nb = (n + 3) // 4
    body = img[3:].view(m, nb)
    g = _gen(seed, 1)
    pick = torch.randint(0, m, (min(m, 1000),), generator=g, device="cuda")
    lut = torch.tensor([2.0, 0.0, 1.0, 0.0], device="cuda")
    q = body[pick].long()
    z = torch.stack([lut[(q >> s) & 3] for s in (0, 2, 4, 6)], 2).reshape(len(pick), 4 * nb)[:, :n]
    z = (z - z.mean(1, keepdim=True)) / z.std(1, keepdim=True).clamp_min(1e-3)
    v = z.T.double() @ torch.randn(len(pick), k, generator=g, device="cuda", dtype=torch.float64)
    v = (v - v.mean(0)) / v.std(0)
    return v.cpu().numpy()


def _vectors(case, seed):
    """Weights, variance components and the drop-ins' vectors, in the FP32 the R driver hands over."""
    n = case["n"]
    X = np.column_stack([np.ones(n), _normal(n, seed, 2, 2)])
    lin = 0.5 * X[:, 1] - 0.4 * X[:, 2]
    if case["call"] in ("ai_q", "trace", "product", "solve", "build"):
        w, tau = np.ones(n), np.array([0.6, 0.4])
        Y = lin + _normal(n, seed, 3)[:, 0]
    else:
        mu = 1 / (1 + np.exp(1.6 - lin))
        w, tau = mu * (1 - mu), np.array([1.0, 0.3])
        y = (torch.rand(n, generator=_gen(seed, 4), device="cuda", dtype=torch.float64).cpu().numpy() < mu)
        Y = np.log(mu / (1 - mu)) + (y - mu) / w
    # stand-ins of the solved vectors an AI step is handed: the diagonal part of Sigma^-1
    d = tau[0] / w + tau[1]
    SX = X / d[:, None]
    f = np.float32
    return dict(Y=Y.astype(f), X=np.asfortranarray(X, dtype=f), w=w.astype(f), tau=tau.astype(f),
                SY=(Y / d).astype(f), SX=np.asfortranarray(SX, dtype=f), cov=np.linalg.inv(X.T @ SX).astype(f))


def _phenotypes(case, img, seed):
    """Half binary, half quantitative phenotypes, each on its own 60-95% of the samples."""
    n, m, k = case["n"], case["m"], case["phenos"]
    gv = _genetic(img, n, m, seed, k)
    rng = np.random.default_rng(int(seed))
    out = []
    for j in range(k):
        C = rng.standard_normal((n, 2))
        mask = np.ones(n, bool)
        mask[rng.permutation(n)[:n * (5 + 35 * j // k) // 100]] = False
        if j % 2 == 0:
            lin = 0.5 * C.sum(1) + np.sqrt(0.5) * gv[:, j]
            y = (rng.uniform(size=n) < 1 / (1 + np.exp(rng.uniform(0.8, 2.2) - lin))).astype(np.float64)
        else:
            h2 = rng.uniform(0.2, 0.6)
            y = 0.3 * C.sum(1) + np.sqrt(h2) * gv[:, j] + np.sqrt(1 - h2) * rng.standard_normal(n)
        trait = "binary" if j % 2 == 0 else "quantitative"
        out.append((trait, mask, prep.make_fit0(y[mask], C[mask], trait)))
    return out


def _chromosomes(m):
    """Two of 22 equal blocks of .bim markers, the first and one in the middle."""
    e = [m * k // 22 for k in range(23)]
    return [(e[0], e[1] - 1), (e[10], e[11] - 1)]


def prepare(case, seed):
    n, m, call = case["n"], case["m"], case["call"]
    img = _bed(n, m, case["miss"], seed, call == "setgeno")
    if call == "setgeno":
        return dict(case=case, ctx=Context(0), bed=img.cpu().numpy())
    ctx = Context(0)
    torch.cuda.synchronize()
    ctx.setgeno_device(img.data_ptr(), img.numel(), n, m)
    s = dict(case=case, ctx=ctx)
    if call == "fits":
        s["specs"] = [serve.FitSpec(f0, trait, mask=mask) for trait, mask, f0 in _phenotypes(case, img, seed)]
    else:
        s.update(_vectors(case, seed))
    del img
    torch.cuda.empty_cache()
    if case["engine"] == "default":
        ctx.grm_build()
    elif case["engine"] == "bf16x3":
        ctx.grm_build(GRM_BF16X3_TC)
        ctx.set_matvec_mode(MV_BF16X3_TC)
    elif case["engine"] == "subset":
        ctx.set_matvec_mode(MV_SUBSET_EXACT)
    return s


# ------------------------------------------------------------------------------------ one pass
def run(s):
    ctx, case = s["ctx"], s["case"]
    call = case["call"]
    if call == "product":
        return ctx.getCrossprodMatAndKin(s["Y"])
    if call == "solve":
        return ctx.getPCG1ofSigmaAndVector(s["w"], s["tau"], s["Y"], MAXITER_PCG, TOL_PCG)
    if call == "coef":
        return ctx.getCoefficients(s["Y"], s["X"], s["w"], s["tau"], MAXITER_PCG, TOL_PCG)
    if call == "loco":
        out = []
        for b, e in _chromosomes(case["m"]):
            ctx.loco_set_bim(b, e)
            out.append(ctx.getCoefficients(s["Y"], s["X"], s["w"], s["tau"], MAXITER_PCG, TOL_PCG))
        ctx.loco_clear()
        return out
    if call == "trace":
        tr, used = ctx.GetTrace_q(s["SX"], s["X"], s["w"], s["tau"], s["cov"], NRUN, MAXITER_PCG, TOL_PCG, CUTOFF,
                                  PROBE_SEED)
        return {"trace": tr, "nrun": used}
    if call in ("ai", "ai_q"):
        fn = ctx.getAIScore if call == "ai" else ctx.getAIScore_q
        return fn(s["Y"], s["X"], s["w"], s["tau"], s["SY"], s["SX"], s["cov"], NRUN, MAXITER_PCG, TOL_PCG, CUTOFF,
                  PROBE_SEED)
    if call == "setgeno":
        ctx.setgeno(s["bed"], case["n"], case["m"])
        return {"freq": ctx.allele_freq(), "invstd": ctx.invstd(), "mac": ctx.mac(), "mask": ctx.qc_marker_mask(),
                "diag": ctx.grm_diag_f32(), "packed": ctx.packed_geno()}
    if call == "grm":
        ctx.grm_build(GRM_FP32_SIMT)
        return ctx.grm_get()
    if call == "build":
        ctx.grm_build(GRM_BF16X3_TC)
        return ctx.getCrossprodMatAndKin(s["Y"])
    # new phenotypes every time: their subsets are set up inside the call
    ctx.engine_forget_subsets()
    res, _ = native.fit_batch(ctx, s["specs"])
    for r in res:
        if isinstance(r, Exception):
            raise r
    # theta, alpha, eta and Y are FP32 vectors where the reference's driver gets them
    return [{k: np.asarray(r[k], np.float32) for k in ("theta", "coefficients", "linear_predictors", "Y")} for r in res]


def work(case):
    """What a pass cannot do without.  A GRM product: the 2-bit genotypes read once, 4 n m FLOPs a
    column; solves are counted at two products (they take three to eight)."""
    n, m, call = case["n"], case["m"], case["call"]
    geno = n * m / 4
    if call == "setgeno":
        return {"bytes": 2 * geno + 4 * n + 13 * m, "flops": 2.0 * n * m}
    if call == "grm":
        return {"bytes": geno + 4.0 * n * n, "flops": float(n) * n * m}
    if call == "build":
        return {"bytes": geno + 4.0 * n * n, "flops": float(n) * n * m}
    passes, cols = {"product": (1, 1), "solve": (2, 1), "coef": (2, 4), "loco": (4, 4), "trace": (2, 45),
                    "ai": (4, 24), "ai_q": (4, 24), "fits": (20, 20)}[call]
    k = case.get("phenos", 1)
    if case["engine"] in ("bf16x3", "default"):  # a resident GRM, half of which says everything
        return {"bytes": passes * 2.0 * n * n + 8.0 * n * cols, "flops": 2.0 * n * n * cols * passes}
    return {"bytes": passes * geno + 8.0 * n * cols * k, "flops": 4.0 * n * m * cols * passes * k}


# ------------------------------------------------------------------------------------ the same in FP64
class _Cohort:
    """setgeno over the samples of ``keep`` (a bool mask, or all) and the product Z (Z' v) / M."""

    def __init__(self, img, n, m, keep=None, drop=None):
        self.n, self.m, self.nb = n, m, (n + 3) // 4
        self.body = img[3:].view(m, self.nb)
        self.keep = np.ones(n, bool) if keep is None else keep
        self.S = torch.from_numpy(np.nonzero(self.keep)[0]).cuda()
        mk = torch.from_numpy(self.keep).cuda()
        count = torch.zeros(m, 4, dtype=torch.int64, device="cuda")
        for i, f in self._fields():
            for v in range(4):
                count[i:i + len(f), v] = ((f == v) & mk).sum(1)
        c = count.cpu().numpy()
        nn, f32 = len(self.S), np.float32
        nmiss, allele = c[:, 1], 2 * c[:, 0] + c[:, 2]
        with np.errstate(divide="ignore", invalid="ignore"):
            a0 = allele.astype(f32) / (2 * (nn - nmiss)).astype(f32)
            fill = np.where(np.isfinite(a0), np.floor((f32(2) * a0).astype(np.float64) + 0.5), 0).astype(np.int64)
        allele = allele + fill * nmiss
        freq = allele.astype(f32) / f32(2 * nn)
        ok = (np.minimum(freq, f32(1) - freq) >= f32(0.01)) & (nmiss.astype(f32) / f32(nn) <= f32(0.15))
        self.mask, self.mac, self.freq = ok, np.minimum(allele, 2 * nn - allele), allele / (2.0 * nn)
        p = self.freq
        sd = np.sqrt(2 * p * (1 - p))
        self.inv = np.where(sd > 0, 1 / np.where(sd > 0, sd, 1), 0)
        use = ok.copy()
        if drop is not None:
            use[drop[0]:drop[1] + 1] = False
        self.M = int(use.sum())
        z = np.stack([(2 - 2 * p), (fill - 2 * p), (1 - 2 * p), (0 - 2 * p)], 1) * (self.inv * use)[:, None]
        self.lut = torch.from_numpy(z).cuda()
        self.diag = self._diag()

    def _fields(self):
        step = max(1, (1 << 27) // (4 * self.nb))
        sh = torch.tensor([0, 2, 4, 6], dtype=torch.uint8, device="cuda")
        for i in range(0, self.m, step):
            q = self.body[i:i + step]
            yield i, ((q[:, :, None] >> sh) & 3).reshape(len(q), -1)[:, :self.n]

    def columns(self):
        """Blocks of standardised genotypes (markers x samples of S)."""
        everyone = len(self.S) == self.n
        for i, f in self._fields():
            z = torch.gather(self.lut[i:i + len(f)], 1, (f if everyone else f[:, self.S]).long())
            yield i, z

    def _diag(self):
        d = torch.zeros(len(self.S), dtype=torch.float64, device="cuda")
        for _, z in self.columns():
            d += (z * z).sum(0)
        return d

    def product(self, V):
        u = torch.zeros_like(V)
        for _, z in self.columns():
            u += z.T @ (z @ V)
        return u / self.M

    def dense(self):
        k = torch.zeros(len(self.S), len(self.S), dtype=torch.float64, device="cuda")
        for _, z in self.columns():
            k += z.T @ z
        return k / self.M


def _pcg(co, w, tau, B):
    """Columns solved together, each stopped at sum r^2 <= tol."""
    w = w[:, None]
    minv = 1 / (tau[1] * co.diag[:, None] / co.M + tau[0] / w).clamp_min(1e-4)
    X, R = torch.zeros_like(B), B.clone()
    Z = minv * R
    P = Z.clone()
    live = torch.nonzero((R * R).sum(0) > TOL_PCG)[:, 0]
    for _ in range(MAXITER_PCG):
        if not len(live):
            break
        p, r, z = P[:, live], R[:, live], Z[:, live]
        ap = tau[0] * p / w + tau[1] * co.product(p)
        rz = (r * z).sum(0)
        a = rz / (p * ap).sum(0)
        X[:, live] += a * p
        r = r - a * ap
        z1 = minv * r
        P[:, live] = z1 + (z1 * r).sum(0) / rz * p
        R[:, live], Z[:, live] = r, z1
        live = live[(r * r).sum(0) > TOL_PCG]
    return X


def _mix(z):
    with np.errstate(over="ignore"):
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _probes(start, end, index):
    """The +-1 probes of the documented counter hash of (seed, run, sample)."""
    idx = index.astype(np.uint64)
    out = []
    with np.errstate(over="ignore"):
        for r in range(start, end):
            h = _mix(np.array([PROBE_SEED], np.uint64) ^ np.uint64(0x5851F42D4C957F2D))
            h = _mix(h ^ (np.array([r], np.uint64) * np.uint64(0x9E3779B97F4A7C15)))
            h = _mix(h ^ (idx * np.uint64(0xD1B54A32D192ED03)))
            out.append(np.where(h >> np.uint64(63) == 1, 1.0, -1.0))
    return torch.from_numpy(np.stack(out, 1)).cuda()


def _cv(x):
    x = np.asarray(x)
    return x.std(ddof=1) / x.mean() / len(x)


def _trace(co, SX, w, tau, cov, quant):
    """(tr P, tr PK, probes used)."""
    t1, t0, start, end = [], [], 0, NRUN
    index = co.S.cpu().numpy()
    while True:
        U = _probes(start, end, index)
        Pu = _pcg(co, w, tau, U)
        Pu = Pu - SX @ (cov @ (SX.T @ U))
        t1 += (co.product(U) * Pu).sum(0).tolist()
        t0 += (U * Pu).sum(0).tolist()
        if not (_cv(t1) > CUTOFF or (quant and _cv(t0) > CUTOFF)):
            return np.mean(t0), np.mean(t1), len(t1)
        start, end = end, end + 10


def _inv_upper(A):
    """The inverse of the symmetric matrix that A's upper triangle says (inv_sympd(symmatu(A)))."""
    return torch.linalg.inv(torch.triu(A) + torch.triu(A, 1).T)


def _coef(co, Y, X, w, tau):
    S = _pcg(co, w, tau, torch.column_stack([Y, X]))
    SY, SX = S[:, 0], S[:, 1:]
    cov = _inv_upper(X.T @ SX)
    alpha = cov @ (SX.T @ Y)
    return dict(Sigma_iY=SY, Sigma_iX=SX, cov=cov, alpha=alpha, eta=Y - tau[0] * (SY - SX @ alpha) / w)


def _ai(co, Y, X, w, tau, SY, SX, cov, quant):
    if quant:
        cov = _inv_upper(X.T @ SX)
    PY = SY - SX @ (cov @ (SX.T @ Y))
    APY = co.product(PY[:, None])[:, 0]
    t0, t1, _ = _trace(co, SX, w, tau, cov, quant)
    S = _pcg(co, w, tau, torch.column_stack([APY, PY] if quant else [APY]))
    Q = S - SX @ (cov @ (SX.T @ S))
    out = dict(YPAPY=float(PY @ APY), PY=PY)
    if not quant:
        return dict(out, Trace=float(t1), AI=float(APY @ Q[:, 0]))
    c = float(PY @ Q[:, 0])
    return dict(out, YPA0PY=float(PY @ PY), Trace=np.array([t0, t1]),
                AI=np.array([[float(PY @ Q[:, 1]), c], [c, float(APY @ Q[:, 0])]]))


class _Dense:
    """A cohort with its GRM formed, for whole fits."""

    def __init__(self, co):
        self.K, self.diag, self.M, self.S = co.dense(), co.diag, co.M, co.S

    def product(self, V):
        return self.K @ V


def _fit(co, trait, f0, tol=0.02, maxiter=20):
    """glmmkin.ai_PCG_Rcpp_Binary / _Quantitative from the reference's fit0."""
    binary = trait == "binary"
    y, X, off, eta, alpha = (torch.from_numpy(np.ascontiguousarray(f0[k], dtype=np.float64)).cuda() for k in (
        "y", "X", "offset", "linear_predictors", "coefficients"))
    n = len(y)

    def working(eta):
        if not binary:
            return y - off, torch.ones_like(y)
        mu = 1 / (1 + torch.exp(-eta))
        v = mu * (1 - mu)
        return eta - off + (y - mu) / v, v

    def get_coef(tau, alpha0, eta0):
        Y, W = working(eta0)
        for _ in range(maxiter):
            rc = _coef(co, Y, X, W, tau)
            eta = rc["eta"] + off
            Y, W = working(eta)
            a = rc["alpha"]
            done = float(((a - alpha0).abs() / (a.abs() + alpha0.abs() + 0.1)).max()) < 0.1
            alpha0 = a
            if done:
                break
        return dict(rc, Y=Y, W=W, eta=eta)

    def score(rc, tau):
        return _ai(co, rc["Y"], X, rc["W"], tau, rc["Sigma_iY"], rc["Sigma_iX"], rc["cov"], not binary)

    def newton(rc, tau0):
        re = score(rc, tau0)
        if binary:
            d = np.array([0.0, (re["YPAPY"] - re["Trace"]) / re["AI"]])
            zero = np.array([True, True])
        else:
            d = np.linalg.solve(re["AI"], np.array([re["YPA0PY"] - re["Trace"][0], re["YPAPY"] - re["Trace"][1]]))
            zero = tau0 < tol
        t = tau0 + d
        t[zero & (t < tol)] = 0
        step = 1.0
        while (t < 0).any():
            step *= 0.5
            t = tau0 + step * d
            if not binary:
                t[zero & (t < tol)] = 0
        t[t < tol] = 0
        return t

    tau = np.array([1.0, 0.1 if binary else 0.0])
    rc = get_coef(tau, alpha, eta)
    re = score(rc, tau)
    if binary:
        tau = np.array([1.0, max(0.0, tau[1] + tau[1] ** 2 * (re["YPAPY"] - re["Trace"]) / n)])
    else:
        tau = np.array([max(0.0, tau[0] + tau[0] ** 2 * (re["YPA0PY"] - re["Trace"][0]) / n),
                        max(0.0, tau[1] + tau[1] ** 2 * (re["YPAPY"] - re["Trace"][1]) / n)])
    for _ in range(maxiter):
        tau0 = tau
        rc = get_coef(tau, rc["alpha"] if binary else alpha, eta)
        tau = newton(rc, tau0)
        alpha, eta = rc["alpha"], rc["eta"]
        if tau[1] <= 0 or (np.abs(tau - tau0) / (np.abs(tau) + np.abs(tau0) + tol)).max() < tol:
            break
        if tau.max() > tol ** -2:
            break
    rc = get_coef(tau, alpha, eta)
    return {"theta": tau, "coefficients": rc["alpha"], "linear_predictors": rc["eta"], "Y": rc["Y"]}


def exact(case, seed):
    n, m, call = case["n"], case["m"], case["call"]
    size = float(n) * m
    if size > {"ai": 1.5e9, "ai_q": 1.5e9, "trace": 5.1e9, "fits": 2e7, "coef": 1.6e10, "loco": 5.1e9}.get(call, 1.6e10):
        return None
    img = _bed(n, m, case["miss"], seed, call == "setgeno")
    if call == "fits":
        return [_fit(_Dense(_Cohort(img, n, m, mask)), trait, f0) for trait, mask, f0 in _phenotypes(case, img, seed)]
    if call == "loco":
        cohorts = [_Cohort(img, n, m, drop=r) for r in _chromosomes(m)]
    else:
        co = _Cohort(img, n, m)
    if call == "setgeno":
        ok = co.mask
        return {"freq": co.freq[ok], "invstd": co.inv[ok], "mac": None, "mask": None, "diag": co.diag, "packed": None}
    if call == "grm":
        return co.dense()
    v = {k: torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).cuda() for k, x in _vectors(case, seed).items()}
    tau = v["tau"].tolist()
    if call in ("product", "build"):
        return co.product(v["Y"][:, None])[:, 0]
    if call == "solve":
        return _pcg(co, v["w"], tau, v["Y"][:, None])[:, 0]
    if call == "coef":
        return _coef(co, v["Y"], v["X"], v["w"], tau)
    if call == "loco":
        return [_coef(c, v["Y"], v["X"], v["w"], tau) for c in cohorts]
    if call == "trace":
        t0, t1, _ = _trace(co, v["SX"], v["w"], tau, v["cov"], True)
        return {"trace": np.array([t0, t1]), "nrun": None}
    return _ai(co, v["Y"], v["X"], v["w"], tau, v["SY"], v["SX"], v["cov"], call == "ai_q")
