"""Workloads of the engine as a user's program runs them, for timing and comparison.

Every case is one call (or one short run of calls) of the public host API over a seeded synthetic
cohort: whole solves in both forms, the single passes they are made of, restarts, SNP
pre-selection and the learned start.  Sizes are the repository's own cohorts (c1, c2, c4, scaled c3
and c5), test-sized cohorts, and odd sizes around them.  Iteration counts are fixed (relative
tolerance 0), so a case does the same work whatever the solver's path.

A case is a dict of plain values with a "kind":
  solve     init_em, then admixture_qn (Float64, the default form): what run_admixture does once
            the genotypes are on the device
  sweeps    the gradient / Hessian sweeps of both blocks with their results on the host
  em        one EM half-step of each block and the log-likelihood of the current point
  run32     run_admixture(T=Float32), from genotypes to Q and P
  restarts  AdmixBatch: several random starts of several K over one cohort
  skfr      AIM pre-selection (sparse k-means via feature ranking)
  start     the learned start: genotype sketch, encoder forward pass, closed-form P of a given Q
  train     one epoch of the encoder's training (forward, backward, Adam)
"""
from __future__ import annotations

import math

import numpy as np
import torch

import openadmixture_b200 as oa
from openadmixture_b200 import warmstart

SKETCH, PROJ, HIDDEN = 4096, 32, 256        # the shipped encoder's sizes


def listed() -> list[dict]:
    return [
        # test-sized cohort: launches and host round trips count, not arithmetic
        {"name": "solve-tiny", "kind": "solve", "I": 203, "J": 517, "K": 3, "em": 2, "qn": 3, "mode": "ZAL",
         "impute": False, "p_dist": "uniform"},
        # the CPU-sized cohort c1
        {"name": "solve-c1", "kind": "solve", "I": 1000, "J": 10000, "K": 3, "em": 2, "qn": 3, "mode": "ZAL",
         "impute": False, "p_dist": "uniform"},
        # the drop-in cohort c2
        {"name": "solve-c2", "kind": "solve", "I": 10000, "J": 100000, "K": 5, "em": 1, "qn": 1, "mode": "ZAL",
         "impute": False, "p_dist": "uniform"},
        # many clusters and extreme frequencies (c3, scaled down)
        {"name": "solve-k12", "kind": "solve", "I": 20000, "J": 60000, "K": 12, "em": 1, "qn": 1, "mode": "ZAL",
         "impute": False, "p_dist": "beta"},
        # one gradient / Hessian evaluation of each block, ragged sizes, as a program with its own solver takes it
        {"name": "sweeps-k8", "kind": "sweeps", "I": 10003, "J": 40009, "K": 8, "p_dist": "beta"},
        # EM half-steps and a scoring pass on a larger cohort
        {"name": "em-k8", "kind": "em", "I": 20000, "J": 100000, "K": 8, "impute": False, "p_dist": "uniform"},
        # the Float32 form from genotypes to Q and P: the batching cohort's size
        {"name": "run32-c4", "kind": "run32", "I": 20000, "J": 50000, "K": 6, "em": 2, "qn": 3},
        # the Float32 form on the largest cohort here (c5, scaled down)
        {"name": "run32-large", "kind": "run32", "I": 100000, "J": 100000, "K": 8, "em": 1, "qn": 2},
        # choosing K and guarding against local optima
        {"name": "restarts", "kind": "restarts", "I": 2000, "J": 8000, "K": 3, "n": 8, "em": 1, "qn": 2},
        # ancestry-informative SNPs before the likelihood engine (c2)
        {"name": "skfr-c2", "kind": "skfr", "I": 10000, "J": 100000, "K": 5, "s": 10000, "mode": "global", "iters": 8},
        # the learned start at the training cohorts' size
        {"name": "start-k8", "kind": "start", "I": 20000, "J": 100000, "K": 8},
        # two Adam steps at the training batch size
        {"name": "train-k8", "kind": "train", "I": 8192, "J": 10000, "K": 8},
    ]


def _size(rng, lo: int, hi: int) -> int:
    """log-uniform over [lo, hi], odd sizes among them"""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, v | 1 if rng.random() < 0.6 else v & ~7))


def draw(rng) -> dict:
    kind = rng.choice(["solve", "solve", "solve", "sweeps", "em", "run32", "restarts", "skfr", "start", "train"])
    if kind == "solve":
        K = rng.randint(2, 12)
        I = _size(rng, 16 * K, 20000)
        J = _size(rng, 100 * K, int(max(200 * K, min(100000, 8e10 / (I * K * K)))))
        return {"kind": kind, "I": I, "J": J, "K": K, "em": rng.randint(0, 2), "qn": rng.randint(1, 2),
                "mode": rng.choice(["ZAL", "ZAL", "LBQN"]), "impute": rng.random() < 0.25,
                "p_dist": rng.choice(["uniform", "beta"])}
    if kind == "sweeps":
        K = rng.randint(1, 16)
        return {"kind": kind, "I": _size(rng, 50, 10000), "J": _size(rng, 100, 20000), "K": K,
                "p_dist": rng.choice(["uniform", "beta"])}
    if kind == "em":
        K = rng.randint(1, 16)
        return {"kind": kind, "I": _size(rng, 50, 20000), "J": _size(rng, 100, 50000), "K": K,
                "impute": rng.random() < 0.25, "p_dist": rng.choice(["uniform", "beta"])}
    if kind == "run32":
        K = rng.randint(2, 12)
        return {"kind": kind, "I": _size(rng, 40 * K, 40000), "J": _size(rng, 400 * K, 60000), "K": K,
                "em": rng.randint(1, 2), "qn": rng.randint(1, 2)}
    if kind == "restarts":
        K = rng.randint(2, 6)
        return {"kind": kind, "I": _size(rng, 200, 2000), "J": _size(rng, 1000, 8000), "K": K, "n": rng.randint(2, 8),
                "em": 1, "qn": rng.randint(1, 2)}
    if kind == "skfr":
        K = rng.randint(2, 8)
        J = _size(rng, 2000, 80000)
        return {"kind": kind, "I": _size(rng, 300, 10000), "J": J, "K": K, "s": max(64, J // rng.randint(5, 40)),
                "mode": rng.choice(["global", "local"]), "iters": rng.randint(3, 8)}
    if kind == "start":
        return {"kind": kind, "I": _size(rng, 500, 20000), "J": _size(rng, 8000, 100000), "K": rng.randint(2, 12)}
    return {"kind": kind, "I": _size(rng, 1000, 8192), "J": 10000, "K": rng.randint(2, 12)}


def _spec(case, seed):
    beta = case.get("p_dist") == "beta"
    return oa.CohortSpec("case", case["I"], case["J"], case["K"], alpha=0.5, p_dist="beta" if beta else "uniform",
                         p_lo=1e-3 if beta else 0.05, p_hi=1 - 1e-3 if beta else 0.95, miss=0.01, seed=seed)


def _point(case, seed, q_true, p_true):
    """A point such as the solver visits: near the cohort's Q and P, inside the projections' bounds."""
    rng = np.random.default_rng(seed)
    q = 0.8 * q_true + 0.2 * rng.dirichlet(np.ones(case["K"]), case["I"])
    q = np.maximum(q, 1e-5)
    q /= q.sum(1, keepdims=True)
    p = np.clip(p_true + rng.normal(0, 0.02, p_true.shape), 1e-5, 1 - 1e-5)
    return np.ascontiguousarray(np.concatenate([q, p]))


def _restart_ks(case) -> list[int]:
    return [case["K"] + m % 3 for m in range(case["n"])]


def prepare(case, seed):
    spec = _spec(case, seed)
    q_true, p_true = oa.truth(spec)
    g = oa.genotypes_device(spec, q_true, p_true)
    kind, K = case["kind"], case["K"]
    st = {"case": case, "seed": seed, "g": g}
    if kind in ("solve", "sweeps", "em"):
        d = oa.AdmixData(g.I, g.J, K, 3, skipmissing=not case.get("impute", False), rng=seed)
        st["d"] = d
        st["h"], _ = oa._cu_admixture_base(d, g, g.I, g.J)
        if kind == "solve":
            st["x0"] = d.x.copy()
        else:
            d.x[:] = _point(case, seed, q_true, p_true)
            st["h"].upload(oa.X, d.x)
    elif kind == "restarts":
        ks = _restart_ks(case)
        st["b"] = oa.AdmixBatch(g, ks, seeds=[seed + m for m in range(len(ks))])
        st["x0"] = [oa.init_x(g.I, g.J, k, seed + m) for m, k in enumerate(ks)]
    elif kind == "start":
        S = min(SKETCH, g.J // 2)
        snps = warmstart.sketch_snps(g.J, S, seed)
        st["snps"] = snps
        st["model"] = warmstart.WarmStartMLP(S, PROJ, K, HIDDEN, seed=seed, snps=snps)
        st["q"] = q_true
    elif kind == "train":
        snps = warmstart.sketch_snps(g.J, SKETCH, seed)
        model = warmstart.WarmStartMLP(SKETCH, PROJ, K, HIDDEN, seed=seed, snps=snps)
        st["model"] = model
        st["p0"] = {k: v.clone() for k, v in model.p.items()}
        st["data"] = [(warmstart.sketch(g, snps, PROJ), torch.from_numpy(q_true).to(g.data.device))]
    return st


def run(st):
    case, g = st["case"], st["g"]
    kind, K = case["kind"], case["K"]
    if kind == "solve":
        d, h = st["d"], st["h"]
        d.x[:] = st["x0"]
        d.ll_new = math.nan
        if case["em"] > 0:
            oa.init_em(d, g, case["em"], d_cu=h, g_cu=h, quiet=True)
        oa.admixture_qn(d, g, case["qn"], 0.0, d_cu=h, g_cu=h, mode=case["mode"], quiet=True)
        return {"x": d.x, "ll": d.ll_new}
    if kind == "sweeps":
        h = st["h"]
        Hq, zq = h.grad_hess_q(oa.X, oa.X)
        Hp, zp = h.grad_hess_p(oa.X, oa.X)
        return {"Hq": Hq, "zq": zq, "Hp": Hp, "zp": zp}
    if kind == "em":
        h = st["h"]
        oa.em_q(h, h)
        oa.em_p(h, h)
        return {"x": h.download(oa.X_NEXT), "ll": oa.loglikelihood(h, h)}
    if kind == "run32":
        d, _, _ = oa.run_admixture(g, K, T=np.float32, rng=st["seed"], admix_n_em_iters=case["em"],
                                   admix_n_iter=case["qn"], admix_rtol=0.0, quiet=True)
        return {"q": d.q, "p": d.p}
    if kind == "restarts":
        b = st["b"]
        for mem, x0 in zip(b.members, st["x0"]):
            mem.upload(oa.X, x0)
        b.init_em(case["em"])
        rec = b.run_qn(case["qn"], 0.0)
        return {"ll": rec["ll"], "x": [b.x(m) for m in range(len(b))]}
    if kind == "skfr":
        clusters, aims, objective, iters = oa.skfr(g, K, case["s"], mode=case["mode"], max_iter=case["iters"],
                                                   rng=st["seed"])
        aim = np.zeros(g.J, dtype=np.uint8)          # which SNPs were selected (how many varies in local mode)
        aim[aims] = 1
        return {"clusters": clusters, "aim": aim, "objective": objective, "iters": iters}
    if kind == "start":
        sk = warmstart.sketch(g, st["snps"], PROJ)
        probs = st["model"].forward(sk)
        p = warmstart.warm_p(g, st["q"])
        return {"dos": sk.dos, "freq": sk.freq, "proj": sk.proj, "probs": probs, "p": p}
    model = st["model"]
    for k, v in st["p0"].items():
        model.p[k].copy_(v)
    loss = warmstart.train(model, st["data"], epochs=1, batch=4096, seed=st["seed"])
    return {"loss": np.asarray(loss, dtype=np.float32), "params": dict(model.p)}


def work(case) -> dict:
    I, J, K = case["I"], case["J"], case["K"]
    cells, geno, x = float(I) * J, float((I + 3) // 4) * J, 8.0 * K * (I + J)
    T = K * (K + 1) // 2
    # per cell: qp, then per pass its sums (a multiply and an add each); logarithm or reciprocals as 2
    f_ll, f_emq, f_emp = 2 * K + 4, 2 * K + 4 + 4 * K, 2 * K + 4 + 4 * K
    f_q, f_p = 2 * K + 8 + 4 * (T + K), 2 * K + 8 + 2 * (T + K)
    kind = case["kind"]

    def solve(em, qn):      # EM: both half-steps and a reported log-likelihood; QN: two sweeps of each block, two log-likelihoods
        return {"bytes": em * 3 * (geno + x) + qn * 6 * (geno + x), "flops": cells * (em * (f_emq + f_emp + f_ll) + qn * 2 * (f_q + f_p + f_ll))}

    if kind in ("solve", "run32"):
        return solve(case["em"], case["qn"])
    if kind == "sweeps":
        return {"bytes": 2 * (geno + x) + 8.0 * (I + J) * (K * K + K), "flops": cells * (f_q + f_p)}
    if kind == "em":
        return {"bytes": 3 * (geno + x), "flops": cells * (f_emq + f_emp + f_ll)}
    if kind == "restarts":
        per = [work({**case, "kind": "solve", "K": k}) for k in _restart_ks(case)]
        return {"bytes": sum(w["bytes"] for w in per), "flops": sum(w["flops"] for w in per)}
    if kind == "skfr":      # seeding distances to K centres, then cluster sums and scores on the kept SNPs per iteration
        kept = case["s"] * (K if case["mode"] == "local" else 1)
        return {"bytes": K * geno + case["iters"] * (geno + float((I + 3) // 4) * kept),
                "flops": K * cells + case["iters"] * (cells + float(I) * case["s"] * K)}
    S = min(SKETCH, J // 2)
    D = S + PROJ
    mlp = 2.0 * I * (D * HIDDEN + HIDDEN * HIDDEN + HIDDEN * K)
    if kind == "start":
        return {"bytes": geno + float((I + 3) // 4) * S + float(I) * S + 4.0 * D * HIDDEN + x, "flops": 2.0 * I * S * PROJ + mlp + 4.0 * cells * K}
    return {"bytes": float(I) * S * 2 + 4.0 * 7 * D * HIDDEN, "flops": 3 * mlp - 2.0 * I * D * HIDDEN}


def _dosage(g, j0, j1, mu=None):
    """dosages and non-missing weights of SNPs [j0, j1) as (I, j1 - j0) FP64 tensors"""
    b = g.data[j0:j1]
    c = torch.stack([(b >> (2 * s)) & 3 for s in range(4)], dim=2).reshape(j1 - j0, -1)[:, : g.I].T
    d = torch.where(c >= 2, c - 1, torch.zeros_like(c)).double()
    nm = (c != 1).double()
    if mu is not None:      # a missing dosage is the SNP's mean
        d = torch.where(c == 1, mu[j0:j1][None, :].expand_as(d), d)
        nm = torch.ones_like(nm)
    return d, nm


def exact(case, seed):
    """What run() returns, in 64-bit torch on the device: the single passes and the start's decode, frequencies
    and P.  Whole solves, selections and the network have no such value here."""
    kind, K = case["kind"], case["K"]
    if kind not in ("sweeps", "em", "start"):
        return None
    spec = _spec(case, seed)
    q_true, p_true = oa.truth(spec)
    g = oa.genotypes_device(spec, q_true, p_true)
    I, J, dev = g.I, g.J, g.data.device
    step = max(1, int(4e7) // I)
    if kind == "start":
        S = min(SKETCH, J // 2)
        snps = torch.from_numpy(warmstart.sketch_snps(J, S, seed)).to(dev).long()
        d, nm = _dosage(oa.DeviceGenotypes(g.data[snps].contiguous(), I, S), 0, S)
        freq = d.sum(0) / (2 * nm.sum(0))
        dos = torch.where(nm > 0, d, torch.full_like(d, 3.0)).to(torch.int8)
        q = torch.from_numpy(q_true).to(dev)
        p = torch.empty((J, K), dtype=torch.float64, device=dev)
        for j0 in range(0, J, step):
            d, nm = _dosage(g, j0, min(J, j0 + step))
            p[j0: j0 + step] = (d.T @ q) / (2 * (nm.T @ q))
        return {"dos": dos, "freq": freq, "proj": None, "probs": None, "p": p.clamp(1e-5, 1 - 1e-5)}
    x = torch.from_numpy(_point(case, seed, q_true, p_true)).to(dev)
    q, p = x[:I], x[I:]
    mu = None
    if case.get("impute", False):
        mu = torch.empty(J, dtype=torch.float64, device=dev)
        for j0 in range(0, J, step):
            d, nm = _dosage(g, j0, min(J, j0 + step))
            mu[j0: j0 + step] = d.sum(0) / nm.sum(0)
    iu = torch.triu_indices(K, K, device=dev)
    Hq = torch.zeros((I, len(iu[0])), dtype=torch.float64, device=dev)
    zq = torch.zeros((I, K), dtype=torch.float64, device=dev)
    Hp = torch.zeros((J, len(iu[0])), dtype=torch.float64, device=dev)
    zp = torch.zeros((J, K), dtype=torch.float64, device=dev)
    p_next, ll = torch.zeros((J, K), dtype=torch.float64, device=dev), 0.0
    for j0 in range(0, J, step):
        j1 = min(J, j0 + step)
        d, nm = _dosage(g, j0, j1, mu)
        pj = p[j0:j1]
        qp = q @ pj.T
        om = 1 - qp
        z1, z2 = nm * d / qp, nm * (2 - d) / om
        zq += z1 @ pj + z2 @ (1 - pj)
        if kind == "em":
            ll += float((nm * (d * qp.log() + (2 - d) * om.log())).sum())
            a, b = pj * (z1.T @ q), (1 - pj) * (z2.T @ q)
            p_next[j0:j1] = a / (a + b)
        else:
            w1, w2 = z1 / qp, z2 / om
            Hq += w1 @ (pj[:, iu[0]] * pj[:, iu[1]]) + w2 @ ((1 - pj[:, iu[0]]) * (1 - pj[:, iu[1]]))
            Hp[j0:j1] = (w1 + w2).T @ (q[:, iu[0]] * q[:, iu[1]])
            zp[j0:j1] = (z1 - z2).T @ q
    if kind == "em":
        return {"x": torch.cat([q * zq / (2 * J), p_next]), "ll": ll}

    def full(t):
        m = torch.empty((t.shape[0], K, K), dtype=torch.float64, device=dev)
        m[:, iu[0], iu[1]] = t
        m[:, iu[1], iu[0]] = t
        return m

    return {"Hq": full(Hq), "zq": zq, "Hp": full(Hp), "zp": zp}
