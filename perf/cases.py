"""The work that a user of this framework has it do, as cases that can be timed and checked.

Every case goes through the Python mirror of the C ABI (slemm_gb300.api): the operators of the
Lanczos solvers at their precisions, the REML drivers, the REML gradient, prediction, the GWAS steps
and the loading of a .bed with its marker quality control.  `exact` restates each of them in plain
64-bit torch and numpy.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from slemm_gb300 import _lib, api

_OPS = {"quadform": _lib.OP_QUADFORM, "ldet": _lib.OP_LDET, "matvec": _lib.OP_MATVEC,
        "rmatvec": _lib.OP_RMATVEC, "wrmatvec": _lib.OP_WRMATVEC}
_PRECS = {"fp32": _lib.PREC_FP32, "bf16x2": _lib.PREC_BF16X2, "bf16x3": _lib.PREC_BF16X3,
          "fp16x2": _lib.PREC_FP16X2}
_TAU0 = float(np.float32(3.0) / np.float32(7.0))   # (1 − s2max)/s2max at the default s2max = 0.7


def listed():
    return [
        # one step of a DF-REML fit on a small cohort (2,000 × 10,000, 30 probes and y, two
        # covariates): latency and launches count
        {"name": "op_small", "kind": "op", "op": "quadform", "n": 2000, "m": 10000, "k": 31, "c": 2,
         "prec": "fp16x2", "weighted": False},
        # the same step at the batched workload's size: [y | intercept | 64 probes]
        {"name": "op_block", "kind": "op", "op": "ldet", "n": 100000, "m": 50000, "k": 66, "c": 1,
         "prec": "fp16x2", "weighted": False},
        # and at the window-weighted workload's size, the largest
        {"name": "op_large", "kind": "op", "op": "ldet", "n": 500000, "m": 60000, "k": 66, "c": 1,
         "prec": "fp16x2", "weighted": False},
        # the transposed product of an MC-REML criterion (y and three Monte-Carlo samples), odd sizes
        {"name": "op_narrow", "kind": "op", "op": "rmatvec", "n": 200003, "m": 50021, "k": 4, "c": 1,
         "prec": "fp16x2", "weighted": False},
        # the plain FP32 option (--gpu_precision fp32), one vector, residual weights
        {"name": "op_fp32", "kind": "op", "op": "ldet", "n": 100000, "m": 20000, "k": 1, "c": 1,
         "prec": "fp32", "weighted": True},
        # a whole `--reml` fit: MC-REML, BLUP and BLUE
        {"name": "mc_reml", "kind": "mc_reml", "n": 50000, "m": 20000, "c": 3, "n_MC": 3, "weighted": False},
        # the backward direction: one step on the window weights with the REML gradient
        {"name": "gradient", "kind": "gradient", "n": 50000, "m": 25000, "c": 2, "n_V": 30, "window": 50,
         "weighted": False},
        # `--pred`: genetic values of every individual from the SNP effects
        {"name": "gebv", "kind": "gebv", "n": 100000, "m": 50000},
        # GWAS step 2 by GRAMMAR-Gamma, residual weights in use
        {"name": "score_terms", "kind": "score", "n": 100000, "m": 50000, "c": 3, "weighted": True},
        # GWAS step 2 by windowed MLMA
        {"name": "gwa_windows", "kind": "gwa", "n": 50021, "m": 20011, "c": 2, "n_model": 4000, "block": 1000,
         "weighted": False},
        # GWAS step 1 (`--lmm`): the .gstat.txt quadratic forms
        {"name": "lmm_quadforms", "kind": "lmm", "n": 50000, "m": 20000, "c": 2, "num_qf": 30, "window": 1000,
         "weighted": False},
        # a .bed read from host rows, 5 % of the individuals left out, with MAF and HWE of its markers
        {"name": "load_qc", "kind": "load", "n": 100003, "m": 20011, "keep": 0.95},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["op", "op", "op", "mc_reml", "gradient", "gebv", "score", "gwa", "lmm", "load"])
    weighted = rng.random() < 0.4
    if kind == "op":
        prec = rng.choice(["fp16x2", "fp16x2", "fp16x2", "bf16x2", "bf16x3", "fp32"])
        k = _log(rng, 1, 8 if prec == "fp32" else 130)
        return {"kind": kind, "op": rng.choice(list(_OPS)), "n": _log(rng, 1000, 300000 if k <= 66 else 100000),
                "m": _log(rng, 500, 60000), "k": k, "c": rng.randint(1, 5), "prec": prec, "weighted": weighted}
    if kind == "mc_reml":
        n = _log(rng, 2000, 80000)
        return {"kind": kind, "n": n, "m": _log(rng, 1000, 25000), "c": rng.randint(1, 5),
                "n_MC": max(min(int(4e9 / n ** 2), 30), 3), "weighted": weighted}
    if kind == "gradient":
        return {"kind": kind, "n": _log(rng, 2000, 60000), "m": _log(rng, 2000, 25000), "c": rng.randint(1, 4),
                "n_V": rng.randint(10, 64), "window": rng.choice([20, 50, 101]), "weighted": weighted}
    if kind == "gebv":
        return {"kind": kind, "n": _log(rng, 1000, 300000), "m": _log(rng, 500, 60000)}
    if kind == "score":
        return {"kind": kind, "n": _log(rng, 1000, 200000), "m": _log(rng, 500, 60000), "c": rng.randint(1, 10),
                "weighted": weighted}
    if kind == "gwa":
        m = _log(rng, 2000, 20000)
        return {"kind": kind, "n": _log(rng, 2000, 60000), "m": m, "c": rng.randint(1, 4),
                "n_model": int(m * rng.uniform(0.1, 0.2)), "block": rng.choice([100, 300, 500, 1000]),
                "weighted": weighted}
    if kind == "lmm":
        return {"kind": kind, "n": _log(rng, 2000, 60000), "m": _log(rng, 2000, 20000), "c": rng.randint(1, 4),
                "num_qf": rng.choice([10, 30, 50]), "window": rng.choice([100, 300, 500, 1000]),
                "weighted": weighted}
    return {"kind": "load", "n": _log(rng, 1000, 150000), "m": _log(rng, 500, 30000),
            "keep": rng.choice([1.0, 0.95, 0.8])}


# ---- inputs ------------------------------------------------------------------------------------------
def _bed(n, m, gen, missing=0.0):
    """.bed rows m×ceil(n/4) in device memory: Binomial(2, p_j) counts, p_j ~ U(0.05, 0.5)."""
    nb = (n + 3) // 4
    rows = torch.empty((m, nb), dtype=torch.uint8, device="cuda")
    p = torch.rand(m, generator=gen, device="cuda") * 0.45 + 0.05
    thr = (p * 256).round().to(torch.uint8)
    step = max(1, (1 << 28) // (4 * nb))

    def draws(r):
        words = (r * 4 * nb + 7) // 8
        x = torch.randint(-2 ** 63, 2 ** 63 - 1, (words,), generator=gen, device="cuda", dtype=torch.int64)
        return x.view(torch.uint8)[: r * 4 * nb].view(r, 4 * nb)

    for j0 in range(0, m, step):
        t = thr[j0:j0 + step, None]
        r = t.shape[0]
        code = (draws(r) < t).to(torch.uint8)
        code += (draws(r) < t).to(torch.uint8)
        code += code > 0                        # counts 0, 1, 2 → codes 00, 10, 11
        if missing > 0:
            code[draws(r) < int(missing * 256)] = 1
        code[:, n:] = 0
        code = code.view(r, nb, 4)
        rows[j0:j0 + r] = code[:, :, 0] | (code[:, :, 1] << 2) | (code[:, :, 2] << 4) | (code[:, :, 3] << 6)
    return rows


def _counts(rows, n):
    """Allele-2 counts (a missing call is one copy) of .bed rows, uint8 rows×n."""
    c = torch.stack([(rows >> s) & 3 for s in (0, 2, 4, 6)], dim=2).view(rows.shape[0], -1)[:, :n]
    return (c & 1) + (c >> 1)


def _phenotype(rows, n, gen, h2=0.4):
    m = rows.shape[0]
    idx = torch.randperm(m, generator=gen, device="cuda")[: min(1000, m)]
    beta = torch.randn(idx.numel(), generator=gen, device="cuda") * (h2 / idx.numel()) ** 0.5
    y = torch.randn(n, generator=gen, device="cuda") * (1 - h2) ** 0.5
    for q in range(0, idx.numel(), 200):
        x = _counts(rows[idx[q:q + 200]], n).float()
        x -= x.mean(1, keepdim=True)
        y += beta[q:q + 200] @ (x / x.std(1, keepdim=True).clamp_min(1e-6))
    return y


def _covariates(n, c, gen):
    X = torch.randn((c, n), generator=gen, device="cuda")
    X[0] = 1.0
    return X


def _inputs(case, seed):
    """Everything that is drawn from the seed, as device tensors (columns as rows)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n, m, kind = case["n"], case["m"], case["kind"]
    d = {"rows": _bed(n, m, gen, 0.01)}
    if kind == "load":
        d["keep"] = None
        if case["keep"] < 1.0:
            d["keep"] = torch.nonzero(torch.rand(n, generator=gen, device="cuda") < case["keep"])[:, 0]
        return d
    if kind == "gebv":
        d["alpha"] = torch.randn(m, generator=gen, device="cuda", dtype=torch.float64) / m ** 0.5
        d["flip"] = (torch.rand(m, generator=gen, device="cuda") < 0.5).to(torch.uint8)
        return d
    d["rvec"] = torch.rand(n, generator=gen, device="cuda") * 1.5 + 0.5 if case["weighted"] else None
    d["X"] = _covariates(n, case["c"], gen)
    if kind == "op":
        k, rows_in = case["k"], m if case["op"] == "matvec" else n
        # [y | intercept | normalised Rademacher probes], or SNP effects for the plain product
        if case["op"] == "matvec":
            v = torch.randn((k, m), generator=gen, device="cuda") / m ** 0.5
        else:
            v = torch.randint(0, 2, (k, n), generator=gen, device="cuda").float() * 2 - 1
            v /= n ** 0.5
            v[0] = torch.randn(n, generator=gen, device="cuda")
            if k > 1:
                v[1] = n ** -0.5
        assert v.shape == (k, rows_in)
        d["v"] = v
    else:
        d["y"] = _phenotype(d["rows"], n, gen)   # the GWAS steps take a residual, a fit the trait itself
        if kind in ("mc_reml", "gradient"):
            d["y"] += (torch.randn(case["c"], generator=gen, device="cuda") * 0.5 + 1.0) @ d["X"]
    if kind == "gradient":
        d["wwin"] = torch.rand((m + case["window"] - 1) // case["window"], generator=gen, device="cuda") * 1.9 + 0.1
    if kind == "gwa":
        d["model"] = torch.sort(torch.randperm(m, generator=gen, device="cuda")[: case["n_model"]])[0]
    return d


def _np(t):
    return None if t is None else t.cpu().numpy()


def _orthonormal(X, rvec):
    """Basis of rr∘X (c×n) in FP64, and rr."""
    rr = torch.ones(X.shape[1], dtype=torch.float64, device="cuda") if rvec is None else rvec.double().rsqrt()
    return torch.linalg.qr((X.double() * rr).T)[0].T.contiguous(), rr


def prepare(case, seed):
    """The handle on the packed genotypes, and the call's other arguments as a program has them."""
    api.init(0)
    d, kind = _inputs(case, seed), case["kind"]
    n, m = case["n"], case["m"]
    torch.cuda.synchronize()   # the library reads the inputs on its own stream
    if kind == "load":
        return {"case": case, "rows": _np(d["rows"]), "keep": _np(d["keep"])}
    g = api.Genotypes(d.pop("rows"), n)
    s = {"case": case, "g": g}
    if kind == "gebv":
        return {**s, "alpha": _np(d["alpha"]), "flip": _np(d["flip"])}
    s.update(X=_np(d["X"].T), rvec=_np(d["rvec"]), persnp=np.ones(m, np.float32))
    if kind in ("op", "score", "lmm"):   # as a fit leaves the handle
        gm = (g.counts()[0].astype(np.int32) / np.float32(n)).astype(np.float32)
        w = (1.0 / (gm * (2.0 - gm) / 2.0) / np.float32(m)).astype(np.float32)
        Q, rr = _orthonormal(d["X"], d["rvec"])
        g.set_weights(gm, w, _np(rr.float()) if case["weighted"] else None)
        g.set_projection(_np(Q.float().T))
    if kind == "op":
        g.set_precision(_PRECS[case["prec"]])
        out = torch.empty((case["k"], m if case["op"] in ("rmatvec", "wrmatvec") else n), device="cuda")
        return {**s, "v": d["v"], "out": out}
    s["y"] = _np(d["y"])
    if kind == "gradient":
        s["wwin"] = _np(d["wwin"])
        s["window"] = (np.arange(m) // case["window"]).astype(np.int32)
    if kind == "gwa":
        s["model"] = _np(d["model"])
    return s


_GWA = {"tau": 1.5, "cfactor": 0.97, "snp_var": 0.4, "mac": 20}
_GRAD = {"sigma_g2": 0.2, "sigma_e2": 0.8}   # a first guess, as an optimiser starts from
_LR = 1e-4


def run(state):
    case, g = state["case"], state.get("g")
    kind = case["kind"]
    if kind == "op":
        g.op_device(_OPS[case["op"]], state["v"], state["out"], _TAU0)
        return state["out"]
    if kind == "mc_reml":
        r = g.LMC_REML(state["rvec"], state["X"], state["y"], state["persnp"], seed=7, n_MC=case["n_MC"])
        return {q: r[q] for q in ("vg", "ve", "h2", "Py", "snp_blup", "blue")}
    if kind == "gradient":
        r = g.REML_grad(state["rvec"], state["X"], state["y"], state["persnp"], state["window"], state["wwin"],
                        n_V=case["n_V"], seed=7, **_GRAD)
        # gradients of the window weights in the weights' own type, and the weights one step on
        d_w = r["d_w"].astype(state["wwin"].dtype)
        return {"d_sigma_g2": float(r["d_sigma_g2"]), "d_sigma_e2": float(r["d_sigma_e2"]), "d_w": d_w,
                "wwin": state["wwin"] + np.float32(_LR) * d_w}
    if kind == "gebv":
        return g.gebv(state["alpha"], state["flip"])
    if kind == "score":
        return g.score_terms(state["y"], 20)
    if kind == "gwa":
        r = g.gwa_windows(state["y"], state["rvec"], state["X"], state["model"], 0, case["m"] - 1, case["block"],
                          _GWA["tau"], case["n_model"], _GWA["cfactor"], _GWA["snp_var"], _GWA["mac"])
        return [v.astype(np.float32) for v in r]   # the columns of the statistics table
    if kind == "lmm":
        r = g.LMM_quadforms(state["y"], _TAU0, case["num_qf"], case["window"])
        return {**r, "variants": np.array(r["variants"], np.int64)}
    h = api.Genotypes(state["rows"], case["n"], state["keep"])
    maf, hwep = h.marker_qc()
    counts = h.counts()
    h.close()
    return [maf, hwep, *counts]


def work(case):
    """Bytes: the packed matrix once for each product over it, and each dense input and output once.
    Operations: two for each count and column of a product."""
    n, m, kind = case["n"], case["m"], case["kind"]
    packed = m * ((n + 3) // 4)
    if kind == "op":
        k, passes = case["k"], 2 if case["op"] in ("quadform", "ldet") else 1
        rows = 2 * n if passes == 2 else n + m
        return {"bytes": passes * packed + 4 * k * rows, "flops": passes * 2 * n * m * k}
    if kind == "mc_reml":   # a seed of a few steps and a handful of criterion products
        k, steps, evals = 1 + 2 * case["n_MC"], 4, 4
        return {"bytes": (2 * steps + evals + 3) * packed + 4 * k * n * 2 * steps,
                "flops": 2 * n * m * (2 * steps * k + evals * (1 + case["n_MC"]) + case["n_MC"] + 2)}
    if kind == "gradient":
        k, steps = 1 + case["n_V"], 8
        return {"bytes": (2 * steps + 1) * packed + 4 * k * n * 2 * steps,
                "flops": 2 * n * m * (2 * steps * k + 2 * case["n_V"] + 1)}
    if kind == "gebv":
        return {"bytes": packed + 8 * (m + n), "flops": 2 * n * m}
    if kind == "score":
        return {"bytes": packed + 4 * n * (2 + case["c"]) + 8 * m, "flops": 2 * n * m * (3 + case["c"])}
    if kind == "gwa":
        bs = min(case["block"], case["n_model"] // 2 * 2)
        nb = max(1, 2 * case["n_model"] // bs - 1)
        return {"bytes": 2 * packed + 4 * n * (2 + case["c"]) + 16 * m,
                "flops": nb * (bs * bs * n + bs ** 3 / 3) + 2.0 * m * bs * n + m * bs * bs}
    if kind == "lmm":
        ws, q = min(case["window"], m), case["num_qf"]
        return {"bytes": 12 * packed + 8 * q * n, "flops": q * (ws * ws * n + ws ** 3 / 3) + 20.0 * n * m * q}
    return {"bytes": 2.95 * packed, "flops": 0}


# ---- the same in 64 bits --------------------------------------------------------------------------------
class _Dense:
    """Centred counts as 64-bit blocks of SNP rows, kept when they fit."""

    def __init__(self, rows, n):
        self.rows, self.n, self.m = rows, n, rows.shape[0]
        self.step = max(1, (1 << 30) // n)
        keep = self.m * n * 8 < 30e9
        self.pc = torch.cat([_counts(b, n).sum(1, dtype=torch.int64) for b in rows.split(self.step)])
        self.mean = self.pc.double() / n
        self.kept = [self._make(j) for j in range(0, self.m, self.step)] if keep else None

    def _make(self, j):
        return _counts(self.rows[j:j + self.step], self.n).double() - self.mean[j:j + self.step, None]

    def blocks(self):
        for q, j in enumerate(range(0, self.m, self.step)):
            yield j, self.kept[q] if self.kept else self._make(j)

    def some(self, idx):
        return _counts(self.rows[idx], self.n).double() - self.mean[idx, None]

    def t(self, u):   # columns as rows: (k, n) → (k, m)
        return torch.cat([u @ z.T for _, z in self.blocks()], dim=1)

    def z(self, v):   # (k, m) → (k, n)
        return sum(v[:, j:j + z.shape[0]] @ z for j, z in self.blocks())

    def zwzt(self, u, w):
        return sum(((u @ z.T) * w[j:j + z.shape[0]]) @ z for j, z in self.blocks())


def _project(Q, v):
    return v - (v @ Q.T) @ Q


def _h0(Z, Q, rr, w, tau, v, projected):
    a = rr * Z.zwzt(rr * (_project(Q, v) if projected else v), w)
    return (_project(Q, a) if projected else a) + tau * v


def _cg(apply, B, tol, most, groups=None):
    """Conjugate gradients on every row of B at once; a group of rows stops together when its largest
    relative residual is at most tol.  Returns X and the steps of each group."""
    groups = groups or [B.shape[0]]
    X, R = torch.zeros_like(B), B.clone()
    P, rs, b = R.clone(), (R * R).sum(1), B.norm(dim=1)
    edge = np.cumsum([0] + groups)
    steps = [0] * len(groups)
    live = torch.ones(B.shape[0], dtype=torch.bool, device=B.device)
    for j in range(1, max(most) + 1):
        A = apply(P)
        step = torch.where(live, rs / (P * A).sum(1), 0.0)[:, None]
        X += step * P
        R = R - step * A
        new = (R * R).sum(1)
        res = new.sqrt() / b
        for q in range(len(groups)):
            at = slice(edge[q], edge[q + 1])
            if not steps[q] and (float(res[at].max()) <= tol or j >= most[q]):
                steps[q] = j
                live[at] = False
        if all(steps):
            break
        P = R + (new / rs)[:, None] * P
        rs = new
    return X, [s or j for s in steps]


def _seed_and_solve(H, tau0, B, tol, groups=None):
    """The framework's seed at tau0 (its step counts) and solve(σ) with at most these steps."""
    _, J = _cg(lambda v: H(tau0, v), B, tol, [599] * len(groups or [0]), groups)
    return lambda sigma: _cg(lambda v: H(tau0 + sigma, v), B, 1e-6, J, groups)[0]


def _normals(seed, count):
    """libstdc++'s std::normal_distribution<float> over std::mt19937(seed): Marsaglia's polar method."""
    rs, got, f = np.random.RandomState(seed), [], np.float32
    have = 0
    while have < count:
        u = rs.randint(0, 2 ** 32, size=2 * ((count - have) * 2 // 3 + 64), dtype=np.uint32)
        u = np.minimum(u.astype(f) * f(2.0 ** -32), np.nextafter(f(1), f(0)))
        xy = (2.0 * u.astype(np.float64) - 1.0).astype(f).reshape(-1, 2)
        r2 = xy[:, 0] * xy[:, 0] + xy[:, 1] * xy[:, 1]
        ok = (r2 <= 1.0) & (r2 != 0.0)
        mult = np.sqrt(f(-2.0) * np.log(r2[ok]) / r2[ok])
        got.append((xy[ok][:, ::-1] * mult[:, None]).reshape(-1))
        have += got[-1].size
    return np.concatenate(got)[:count]


def _fit_terms(d, case):
    Z = _Dense(d["rows"], case["n"])
    Q, rr = _orthonormal(d["X"], d["rvec"])
    w = 1.0 / (Z.mean * (2.0 - Z.mean) / 2.0) / case["m"]
    return Z, Q, rr, w


def _exact_op(d, case):
    Z, Q, rr, w = _fit_terms(d, case)
    op, v = case["op"], d["v"].double()
    if op == "matvec":
        return Z.z(v)
    if op in ("rmatvec", "wrmatvec"):
        return Z.t(v) * (w if op == "wrmatvec" else 1.0)
    return _h0(Z, Q, rr, w, _TAU0, v, op == "quadform")


def _exact_mc_reml(d, case):
    n, m, k = case["n"], case["m"], case["n_MC"]
    Z, Q, rr, w = _fit_terms(d, case)
    z = torch.from_numpy(_normals(7 + 54321, (m + n) * k)).cuda().double()
    u, e = z[: m * k].view(k, m), z[m * k:].view(k, n)
    y = d["y"].double()
    V = _project(Q, torch.cat([rr * y[None], rr * Z.z(u * w.sqrt()), e]))
    solve = _seed_and_solve(lambda t, v: _h0(Z, Q, rr, w, t, v, True), _TAU0, V, 5e-3)

    def first_order(s2):
        tau = (1 - s2) / s2
        PV = solve(tau - _TAU0)
        Py = PV[: 1 + k].clone()
        Py[1:] += math.sqrt(tau) * PV[1 + k:]
        Py = _project(Q, Py)
        es = Py.square().sum(1)
        Py = Py * rr
        us = (Z.t(Py) * w.sqrt()).square().sum(1)
        return float(((us[0] / es[0]) / (us[1:].sum() / es[1:].sum())).log()), Py[0]

    s2 = 0.35
    lt1 = math.log((1 - s2) / s2)
    f1, _ = first_order(s2)
    s2 = 0.175 if f1 < 0 else 0.7
    lt2 = math.log((1 - s2) / s2)
    f2, Py = first_order(s2)
    for _ in range(3, 10):
        lt = max(-9.0, min(9.0, (lt1 * f2 - lt2 * f1) / (f2 - f1)))
        if abs(lt - lt2) < 0.002:
            break
        s2 = 1 / (math.exp(lt) + 1)
        f1, (f2, Py) = f2, first_order(s2)
        lt1, lt2 = lt2, lt
    vg = float(y @ Py) / (n - case["c"])
    tau = (1 - s2) / s2
    blup = w * Z.t(Py[None])[0]
    R = 1.0 / rr ** 2
    X = d["X"].double()
    blue = torch.linalg.solve(X @ X.T, X @ (y - Z.z(blup[None])[0] - tau * R * Py))
    return {"vg": vg, "ve": tau * vg, "h2": s2, "Py": Py, "snp_blup": blup, "blue": blue}


def _exact_gradient(d, case):
    n, m, k = case["n"], case["m"], case["n_V"]
    Z, Q, rr, gw = _fit_terms(d, case)
    sg, se = _GRAD["sigma_g2"], _GRAD["sigma_e2"]
    win = torch.arange(m, device="cuda") // case["window"]
    W = gw * d["wwin"].double()[win]
    draws = np.random.RandomState(7 + 54321).randint(0, 2 ** 32, size=n * k, dtype=np.uint32).astype(np.float32)
    V = torch.from_numpy(np.where(draws < np.float32(2.0 ** 31), -1.0, 1.0).reshape(k, n)).cuda() / math.sqrt(n)
    B = _project(Q, torch.cat([rr * d["y"].double()[None], V]))
    H = lambda t, v: _h0(Z, Q, rr, W, t, v, True)   # noqa: E731
    P = _project(Q, _seed_and_solve(H, se / sg, B, 1e-6, [1, k])(0.0))
    T, TV = Z.t(rr * P), Z.t(rr * V)
    a, b = T[0].square(), (T[1:] * TV).sum(0) * (n / k)
    trP, pyy = float((V * P[1:]).sum()) * n / k, float(P[0].square().sum())
    d_w = torch.zeros(d["wwin"].numel(), dtype=torch.float64, device="cuda").index_add_(0, win, gw * (b - a / sg)) * -0.5
    return {"d_sigma_g2": -0.5 * float((W * b).sum() / sg - (W * a).sum() / sg ** 2),
            "d_sigma_e2": -0.5 * (trP / sg - pyy / sg ** 2), "d_w": d_w, "wwin": d["wwin"].double() + _LR * d_w}


def _exact_gebv(d, case):
    out = torch.zeros(case["n"], dtype=torch.float64, device="cuda")
    for rows, al, fl in zip(d["rows"].split(2000), d["alpha"].split(2000), d["flip"].split(2000)):
        x = _counts(rows, case["n"]).double()
        out += torch.where(fl.bool(), -al, al) @ x + 2.0 * al[fl.bool()].sum()
    return out


def _exact_score(d, case):
    n = case["n"]
    Q, rr = _orthonormal(d["X"], d["rvec"])
    y, xy, xx = d["y"].double(), [], []
    for rows in d["rows"].split(2000):
        x = 2.0 - _counts(rows, n).double()
        s = x.sum(1)
        x -= s[:, None] / n
        drop = (s <= 20) | (2 * n - s <= 20)
        t = x * rr
        xy.append(torch.where(drop, math.nan, x @ y))
        xx.append(torch.where(drop, math.nan, t.square().sum(1) - (t @ Q.T).square().sum(1)))
    return torch.cat(xy), torch.cat(xx)


def _exact_gwa(d, case):
    n, m = case["n"], case["m"]
    Z = _Dense(d["rows"], n)
    Q, rr = _orthonormal(d["X"], d["rvec"])
    y, model = d["y"].double(), d["model"]
    idx = model.tolist()
    bs = case["block"] if case["block"] <= len(idx) else len(idx) // 2 * 2
    half = bs // 2
    start = [i * half for i in range((len(idx) - half) // half)]
    if (len(idx) - half) % half:
        start.append(len(idx) - bs)
    hi = [idx[s + bs - half // 2] for s in start]
    hi[-1] = m
    xy, xx = torch.empty(m, dtype=torch.float64, device="cuda"), torch.empty(m, dtype=torch.float64, device="cuda")
    lo = 0
    for s, h in zip(start, hi):
        at = model[s:s + bs]
        B = _project(Q, Z.some(at) * rr)
        mu = Z.mean[at]
        L = torch.linalg.cholesky(B @ B.T + torch.diag(len(idx) * _GWA["tau"] * (2.0 - mu) * mu / 2.0))
        for j in range(lo, h, 4000):
            x = Z.some(torch.arange(j, min(h, j + 4000), device="cuda"))
            xy[j:j + x.shape[0]] = -(x @ y)
            t = _project(Q, x * rr)
            q = torch.linalg.solve_triangular(L, B @ t.T, upper=False).square().sum(0)
            xx[j:j + x.shape[0]] = (t.square().sum(1) - q) / _GWA["tau"]
        lo = h
    beta = xy / xx * _GWA["cfactor"]
    se = (_GWA["snp_var"] * _GWA["cfactor"] / xx).sqrt()
    chisq = (beta / se).square()
    s = 2 * n - Z.pc
    drop = (s <= _GWA["mac"]) | (2 * n - s <= _GWA["mac"])
    return [torch.where(drop, math.nan, v) for v in (beta, se, chisq, torch.erfc((chisq / 2).sqrt()))]


def _exact_lmm(d, case):
    n, m = case["n"], case["m"]
    Z, Q, rr, w = _fit_terms(d, case)
    gm = (Z.pc.cpu().numpy().astype(np.int32) / np.float32(n)).astype(np.float32)
    var = [j for j in range(m) if gm[j] * np.float32(n) > 20 and (np.float32(2) - gm[j]) * np.float32(n) > 20]
    libc = ctypes.CDLL(None)
    libc.srand(1)
    for i in range(1, len(var)):   # std::random_shuffle on the C library's rand()
        j = libc.rand() % (i + 1)
        var[i], var[j] = var[j], var[i]
    var = var[: case["num_qf"]]
    at = torch.tensor(var, device="cuda")
    x = Z.some(at)
    v = _project(Q, x * rr)
    Px = _seed_and_solve(lambda t, u: _h0(Z, Q, rr, w, t, u, True), _TAU0, v, 5e-4)(0.0)
    ws, xBx = case["window"], []
    for c, j in enumerate(var):
        lo = 0 if j < ws // 2 else m - ws if j > m - ws // 2 else j - ws // 2
        B = _project(Q, Z.some(torch.arange(lo, lo + ws, device="cuda")) * rr)
        z = B @ v[c]
        A = B @ B.T + torch.diag(_TAU0 / w[lo:lo + ws])
        xBx.append((v[c] @ v[c] - z @ torch.linalg.solve(A, z)) / _TAU0)
    return {"xPy": x @ d["y"].double(), "xPx": (v * Px).sum(1), "xBx": torch.stack(xBx), "xSx": v.square().sum(1),
            "variants": None}


def _exact_load(d, case):
    """Exact test of Hardy–Weinberg equilibrium (Wigginton, Cutler and Abecasis, 2005) from log-gammas."""
    maf, hwe = [], []
    for rows in d["rows"].split(1000):
        x = _counts(rows, case["n"])
        x = x if d["keep"] is None else x[:, d["keep"]]
        n = x.shape[1]
        f = x.sum(1, dtype=torch.int64).double() / (2 * n)
        maf.append(torch.minimum(f, 1 - f))
        n1, n2 = (x == 1).sum(1), (x == 2).sum(1)
        rare = torch.minimum(2 * n2 + n1, 2 * (n - n1 - n2) + n1)
        h = (rare % 2)[:, None] + 2 * torch.arange(int(rare.max()) // 2 + 1, device="cuda")
        r = ((rare[:, None] - h) // 2).double()
        ok, h = r >= 0, h.double()
        r = r.clamp_min(0)
        c = (n - h - r).clamp_min(0)
        lp = h * math.log(2.0) - torch.lgamma(r + 1) - torch.lgamma(h + 1) - torch.lgamma(c + 1)
        lp = torch.where(ok, lp, -math.inf)
        obs = torch.gather(lp, 1, ((n1 - rare % 2) // 2)[:, None])
        p = (lp - lp.max(1, keepdim=True)[0]).exp()
        hwe.append((torch.where(lp <= obs + 1e-7, p, 0.0).sum(1) / p.sum(1)).clamp_max(1.0))
    return [torch.cat(maf), torch.cat(hwe), None, None, None, None]


_EXACT = {"op": _exact_op, "mc_reml": _exact_mc_reml, "gradient": _exact_gradient, "gebv": _exact_gebv,
          "score": _exact_score, "gwa": _exact_gwa, "lmm": _exact_lmm, "load": _exact_load}


def exact(case, seed):
    return _EXACT[case["kind"]](_inputs(case, seed), case)
