"""Timed workloads: what a user's program has this framework do, per call.

Families (field "kind"):
  lda         one Gibbs sweep of the topic model (theta, phi, then every
              token's topic), LdaGibbs.sweep
  mixture     one Gibbs sweep of a Gaussian mixture, GmmGibbs.sweep: the
              hierarchical model (weights, means, covariances, labels) or the
              shared-covariance model with conjugate, elliptical-slice or
              Metropolis moves of the means
  chains      iterations of a per-chain HMC or NUTS schedule on a hierarchical
              logistic regression, HlrChains.run
  pass        log density and / or gradient of many chains on one large design
              matrix, HlrbData.logp_grad (one leapfrog step's work)
  group       the same for many model instances of uneven size in one call,
              HlrGroup.logp_grad (one round of grouped NUTS)
  surrogate   the gradient surrogate of HMC: its prediction at all chains'
              positions (one leapfrog step), or a burst of its online training

exact() recomputes a case's floating outputs in 64 bits from the definition
of the model and of the random substreams (Philox4x32-10 counters
(draw, element, iteration, tag) under the seed), with torch and numpy alone.
"""
import math

import numpy as np
import torch

from augurv2_b200.gmm import GmmGibbs
from augurv2_b200.hlr import HlrChains, HlrData
from augurv2_b200.hlrb import HlrbData, HlrGroup, MlpSurrogate
from augurv2_b200.lda import LdaGibbs

DEV = "cuda"
GROUP_D = (16, 64, 256)
BUFFER = 8192      # replay buffer of the surrogate (its default)


def listed():
    return [
        # a toy corpus, as in a first example: every step is launch latency
        {"name": "lda_example", "kind": "lda", "K": 12, "V": 300, "D": 40, "mean_len": 60},
        # a corpus of abstracts: the usual number of topics, 4e5 tokens
        {"name": "lda_abstracts", "kind": "lda", "K": 50, "V": 10000, "D": 2000, "mean_len": 200},
        # more topics than fit the narrow token kernels, fewer but longer documents
        {"name": "lda_many_topics", "kind": "lda", "K": 130, "V": 5003, "D": 611, "mean_len": 310},
        # a small shared-covariance mixture moved by elliptical slices
        {"name": "mixture_slice", "kind": "mixture", "move": "eslice", "N": 6007, "K": 5, "d": 6},
        # a mid-sized hierarchical mixture, dimension not a multiple of four
        {"name": "mixture_mid", "kind": "mixture", "move": "hier", "N": 20011, "K": 7, "d": 13},
        # the hierarchical mixture at benchmark size
        {"name": "mixture_large", "kind": "mixture", "move": "hier", "N": 200000, "K": 16, "d": 32},
        # a single HMC chain on a small regression: the plain use of the reference's sampler
        {"name": "chain_hmc", "kind": "chains", "method": "hmc", "N": 1000, "D": 10, "C": 1, "iters": 10, "dtype": "f32"},
        # parallel NUTS chains on a wider regression with a bf16 design matrix
        {"name": "chains_nuts", "kind": "chains", "method": "nuts", "N": 2003, "D": 41, "C": 48, "iters": 2, "dtype": "bf16"},
        # every leapfrog step of exact-gradient HMC on the large regression
        {"name": "pass_large", "kind": "pass", "mode": "both", "N": 2000000, "D": 512, "C": 256},
        # one round of grouped NUTS: instances from 1e3 to 1e6 rows, 512 chains each
        {"name": "group_uneven", "kind": "group", "n": 24, "n_lo": 1000, "n_hi": 1000000, "C": 512},
        # every leapfrog step of surrogate HMC
        {"name": "surrogate_step", "kind": "surrogate", "mode": "predict", "D": 512, "C": 256},
        # the surrogate's online training between trajectories
        {"name": "surrogate_train", "kind": "surrogate", "mode": "train", "D": 512, "C": 256, "steps": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("lda", "lda", "mixture", "mixture", "chains", "pass", "group", "surrogate"))
    if kind == "lda":
        K = _log_int(rng, 4, 160)
        V = _log_int(rng, 200, 12000)
        return {"kind": kind, "K": K, "V": V, "D": _log_int(rng, 30, 2500), "mean_len": _log_int(rng, 20, 240)}
    if kind == "mixture":
        move = rng.choice(("hier", "hier", "conj", "eslice", "mwg"))
        if move in ("eslice", "mwg"):
            return {"kind": kind, "move": move, "N": _log_int(rng, 500, 20000), "K": rng.randint(2, 10),
                    "d": rng.randint(2, 9)}
        return {"kind": kind, "move": move, "N": _log_int(rng, 1000, 200000), "K": rng.randint(2, 20),
                "d": rng.randint(2, 32)}
    if kind == "chains":
        if rng.random() < 0.5:
            return {"kind": kind, "method": "hmc", "N": _log_int(rng, 200, 5000), "D": rng.randint(3, 28),
                    "C": _log_int(rng, 1, 256), "iters": 10, "dtype": rng.choice(("f32", "bf16"))}
        return {"kind": kind, "method": "nuts", "N": _log_int(rng, 200, 2000), "D": rng.randint(5, 40),
                "C": _log_int(rng, 1, 48), "iters": 2, "dtype": rng.choice(("f32", "bf16"))}
    if kind == "pass":
        return {"kind": kind, "mode": rng.choice(("both", "grad", "logp")), "N": _log_int(rng, 2000, 1500000),
                "D": 8 * _log_int(rng, 2, 64), "C": _log_int(rng, 16, 512)}
    if kind == "group":
        return {"kind": kind, "n": rng.randint(3, 24), "n_lo": _log_int(rng, 300, 2000),
                "n_hi": _log_int(rng, 20000, 400000), "C": rng.randint(32, 512)}
    mode = rng.choice(("predict", "train"))
    c = {"kind": kind, "mode": mode, "D": 8 * _log_int(rng, 2, 64), "C": _log_int(rng, 16, 512)}
    if mode == "train":
        c["steps"] = rng.randint(5, 20)
    return c


# ---- inputs ----------------------------------------------------------------

def _corpus(case, seed):
    """Documents of the generative process (alpha 0.1, beta 0.01) and the
    topics that generated the tokens, one in ten of them replaced: a chain's
    state once it has found the topics.  The documents' lengths belong to the
    case, their contents to the seed."""
    K, V, D = case["K"], case["V"], case["D"]
    lens = np.maximum(1, np.random.default_rng(D).poisson(case["mean_len"], size=D))
    rng = np.random.default_rng([seed, 1])
    off = np.zeros(D + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    T = int(off[-1])
    theta = rng.dirichlet(np.full(K, 0.1), size=D)
    ct = np.cumsum(theta, axis=1)
    doc = np.repeat(np.arange(D), lens)
    z = np.minimum(np.searchsorted((ct + np.arange(D)[:, None]).ravel(), rng.random(T) * ct[doc, -1] + doc) - doc * K, K - 1)
    z = np.maximum(z, 0)
    g = rng.gamma(0.01, size=(K, V)) + 1e-300
    cp = np.cumsum(g / g.sum(1, keepdims=True), axis=1)
    u = rng.random(T)
    w = np.empty(T, np.int64)
    for k in range(K):
        m = z == k
        w[m] = np.minimum(np.searchsorted(cp[k], u[m] * cp[k, -1]), V - 1)
    again = rng.random(T) < 0.1
    z = np.where(again, rng.integers(0, K, T), z)
    return off.astype(np.int32), w.astype(np.int32), z.astype(np.int32)


def _mixture(case, seed):
    """Points of a mixture with well apart means, labels from the generating
    components (one in twenty replaced)."""
    N, K, d = case["N"], case["K"], case["d"]
    rng = np.random.default_rng([seed, 2])
    mus = rng.standard_normal((K, d)) * 5.0
    A = rng.standard_normal((K, d + 2, d))
    covs = np.einsum("kai,kaj->kij", A, A) / (d + 2) + 0.05 * np.eye(d)
    if case["move"] != "hier":
        covs = np.broadcast_to(covs[:1], (K, d, d)).copy()
    pis = rng.dirichlet(np.full(K, 2.0))
    z = rng.choice(K, size=N, p=pis).astype(np.int32)
    L = np.linalg.cholesky(covs)
    Y = rng.standard_normal((N, d))
    for k in range(K):
        m = z == k
        Y[m] = mus[k] + Y[m] @ L[k].T
    again = rng.random(N) < 0.05
    z0 = np.where(again, rng.integers(0, K, N), z).astype(np.int32)
    mu_start = mus + 0.05 * rng.standard_normal((K, d))
    return Y.astype(np.float32), z0, mu_start, covs, pis


def _regression(case, seed):
    N, D = case["N"], case["D"]
    rng = np.random.default_rng([seed, 3])
    X = rng.standard_normal((N, D)).astype(np.float32)
    s2 = float(np.clip(1.0 / rng.gamma(2.0), 0.4, 2.0))
    beta = rng.standard_normal(D) * np.sqrt(s2) * (1.0 if D < 30 else math.sqrt(10.0 / D))
    y = (rng.random(N) < 1.0 / (1.0 + np.exp(-(X @ beta)))).astype(np.int32)
    init = np.zeros((case["C"], D + 2))
    init[:, :D] = beta + 0.02 * rng.standard_normal((case["C"], D))
    init[:, D + 1] = s2
    return X, y, init


def _design(N, D, seed, scale):
    """X ~ N(0, 1) stored in bf16, labels of a logistic model, on the GPU."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    beta = torch.randn(D, generator=g, device=DEV) * scale
    X = torch.empty((N, D), dtype=torch.bfloat16, device=DEV)
    y = torch.empty(N, dtype=torch.int32, device=DEV)
    for s in range(0, N, 1 << 18):
        e = min(N, s + (1 << 18))
        X[s:e] = torch.randn((e - s, D), generator=g, device=DEV).to(torch.bfloat16)
        t = X[s:e].float() @ beta
        y[s:e] = (torch.rand(e - s, generator=g, device=DEV) < torch.sigmoid(t)).to(torch.int32)
    return X, y, beta, g


def _pass_inputs(case, seed):
    D = case["D"]
    X, y, beta, g = _design(case["N"], D, 7919 * seed + 11, min(1.0, 4.0 / math.sqrt(D)))
    theta = beta + 0.01 * torch.randn((case["C"], D), generator=g, device=DEV)
    return X, y, theta.contiguous()


def _group_sizes(case):
    """Row counts spread over the range on a log scale, made odd and ragged;
    the widths take turns."""
    n, lo, hi = case["n"], case["n_lo"], case["n_hi"]
    return [(int(lo * (hi / lo) ** (i / max(1, n - 1))) + (37 * i) % 101, GROUP_D[(i * 5) % 3]) for i in range(n)]


def _group_inputs(case, seed):
    for i, (N, D) in enumerate(_group_sizes(case)):
        X, y, beta, g = _design(N, D, 7919 * seed + 101 * i + 13, 0.5 if D < 100 else 0.25)
        yield X, y, (beta + 0.01 * torch.randn((case["C"], D), generator=g, device=DEV)).contiguous()


def _pairs(case, seed):
    """Positions around a mode and gradients there: a correlated linear force
    and a mild curvature."""
    D = case["D"]
    g = torch.Generator(device=DEV)
    g.manual_seed(7919 * seed + 17)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    centre, spread = r(D), 0.02 * (0.5 + torch.rand(D, generator=g, device=DEV))
    B = r(D, D) / math.sqrt(D)
    H = 40.0 * (B @ B.T + torch.eye(D, device=DEV))

    def grad(th):
        dt = th - centre
        return (-(dt @ H) + 2.0 * torch.tanh(8.0 * dt / spread.mean()) * spread).contiguous()

    buf = (centre + spread * r(BUFFER, D)).contiguous()
    at = (centre + spread * r(case["C"], D)).contiguous()
    return buf, grad(buf), at


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "lda":
        off, w, z = _corpus(case, seed)
        st["s"] = LdaGibbs(case["K"], case["V"], off, w, 0.1, 0.01, seed=seed, z=z)
    elif kind == "mixture":
        Y, z, mu, covs, pis = _mixture(case, seed)
        K, d = case["K"], case["d"]
        if case["move"] == "hier":
            st["s"] = GmmGibbs(Y, K, np.zeros(d), 25.0 * np.eye(d), alpha=np.ones(K), df=d + 2, scale0=np.eye(d),
                               mu=mu, cov=covs, pis=pis, z=z, seed=seed)
        else:
            st["s"] = GmmGibbs(Y, K, np.zeros(d), 25.0 * np.eye(d), pis=pis, covs=covs[0], mu=mu, z=z,
                               move=case["move"], prop_cov=0.01 * np.eye(d), seed=seed)
    elif kind == "chains":
        X, y, init = _regression(case, seed)
        if case["method"] == "hmc":
            data = HlrData(X, y, has_b=False, vprior="invgamma", a0=1.0, s0=1.0, x_dtype=case["dtype"])
            sched = [{"kind": "HMC", "block": ["theta", "v"], "simlen": 0.1, "eps": 0.01}]
        else:
            data = HlrData(X, y, has_b=True, vprior="exponential", lam=1.0, x_dtype=case["dtype"])
            sched = [{"kind": "NUTS", "block": ["v", "b", "theta"], "eps": 0.5 / math.sqrt(0.2 * case["N"]),
                      "max_depth": 5}]
        st["s"] = HlrChains(data, sched, C=case["C"], init=init, seed=seed)
    elif kind == "pass":
        X, y, theta = _pass_inputs(case, seed)
        data = HlrbData(X, y, prior="student_t", nu=3.0, scale=1.0)
        C, D = theta.shape
        st.update(data=data, theta=theta, work=data.workspace(C),
                  logp=torch.empty(C, dtype=torch.float64, device=DEV), grad=torch.empty((C, D), device=DEV),
                  err=torch.zeros(1, dtype=torch.int32, device=DEV))
    elif kind == "group":
        datas, thetas, logps, grads = [], [], [], []
        for X, y, theta in _group_inputs(case, seed):
            datas.append(HlrbData(X, y, prior="normal", var=1.0))
            thetas.append(theta)
            logps.append(torch.empty(theta.shape[0], dtype=torch.float64, device=DEV))
            grads.append(torch.empty(theta.shape, device=DEV))
        group = HlrGroup(datas, [case["C"]] * len(datas))
        for i in range(len(datas)):
            group.bind(i, thetas[i], logps[i], grads[i])
        group.set_active([True] * len(datas))
        st.update(group=group, datas=datas, thetas=thetas, logps=logps, grads=grads,
                  err=torch.zeros(1, dtype=torch.int32, device=DEV))
    else:
        buf, grad, at = _pairs(case, seed)
        sur = MlpSurrogate(case["D"], seed=seed, device=DEV)
        sur.add(buf, grad)
        sur.refit()
        st.update(sur=sur, at=at, out=torch.empty_like(at))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "lda":
        s = st["s"]
        s.sweep(1)
        return {"theta": s.theta, "phiT": s.phiT, "z": s.z}
    if kind == "mixture":
        s = st["s"]
        s.sweep(1)
        out = {"mu": s.mu, "z": s.z}
        if case["move"] == "hier":
            out.update(pis=s.pis, cov=s.cov)
        return out
    if kind == "chains":
        s = st["s"]
        s.run(case["iters"])
        return {"pars": s.pars, "stats": s.stats}
    if kind == "pass":
        logp, grad = st["data"].logp_grad(st["theta"], case["mode"] != "logp", st["logp"], st["grad"], st["work"],
                                          st["err"], logp=case["mode"] != "grad")
        return {"logp": logp, "grad": grad}
    if kind == "group":
        st["group"].logp_grad(st["err"])
        return {"logp": torch.cat(st["logps"]), "grad": torch.cat([g.view(-1) for g in st["grads"]])}
    sur = st["sur"]
    if case["mode"] == "predict":
        return {"grad": sur.predict(st["at"], st["out"])}
    loss = sur.train(case["steps"])
    return {"loss": loss, "w": sur.w, "m": sur.m, "v": sur.v}


# ---- the work a pass cannot do without -------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "lda":
        K, V, D = case["K"], case["V"], case["D"]
        T = D * case["mean_len"]
        return {"bytes": 4.0 * T + 8.0 * T + 8.0 * D * K + 8.0 * K * V, "flops": 2.0 * K * T + 60.0 * K * (D + V)}
    if kind == "mixture":
        N, K, d = case["N"], case["K"], case["d"]
        flops = 1.0 * K * N * (d * d + 3 * d)
        if case["move"] == "hier":
            flops += 1.0 * N * d * (d + 1) + K * 10.0 * d ** 3
        elif case["move"] != "conj":
            flops += 2.0 * N * (d * d + 3 * d)
        return {"bytes": 4.0 * N * d + 8.0 * N + 16.0 * K * d * (d + 1), "flops": flops}
    if kind == "chains":
        N, D, C = case["N"], case["D"], case["C"]
        evals = case["iters"] * (11 if case["method"] == "hmc" else 4)
        return {"bytes": N * D * (4.0 if case["dtype"] == "f32" else 2.0) + 4.0 * N + 16.0 * C * (D + 2),
                "flops": evals * 4.0 * N * D * C}
    if kind == "pass":
        N, D, C = case["N"], case["D"], case["C"]
        return {"bytes": 2.0 * N * D + 4.0 * N + 8.0 * C * D, "flops": (2.0 if case["mode"] == "logp" else 4.0) * N * D * C}
    if kind == "group":
        C = case["C"]
        b = sum(2.0 * N * D + 4.0 * N + 8.0 * C * D for N, D in _group_sizes(case))
        return {"bytes": b, "flops": sum(4.0 * N * D * C for N, D in _group_sizes(case))}
    D, h = case["D"], 256
    params = 2.0 * D * h + h * h
    if case["mode"] == "predict":
        C = case["C"]
        return {"bytes": 8.0 * C * D + 2.0 * params + 4.0 * D * D, "flops": 2.0 * C * (params + D * D)}
    return {"bytes": case["steps"] * (512 * 8.0 * D + 24.0 * params), "flops": case["steps"] * 6.0 * 512 * params}


# ---- the same in 64 bits ----------------------------------------------------

_M32 = 0xFFFFFFFF


def _philox(pos, elem, it, tag, seed):
    """Philox4x32-10 blocks at counters (pos, elem, it, tag), int64 tensors."""
    pos, elem = torch.broadcast_tensors(torch.as_tensor(pos, device=DEV), torch.as_tensor(elem, device=DEV))
    c = [pos.long() & _M32, elem.long() & _M32, torch.full_like(pos, it).long(), torch.full_like(pos, tag).long()]
    k0, k1 = seed & _M32, (seed >> 32) & _M32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & _M32) ^ c[1] ^ k0, p1 & _M32, ((p0 >> 32) & _M32) ^ c[3] ^ k1, p0 & _M32]
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return c


def _unit(a, b):
    return ((((a & 0xFFFFF) << 32) | b).double() + 0.5) * 2.0 ** -52


def _uniform(pos, elem, it, tag, seed):
    c = _philox(pos, elem, it, tag, seed)
    return _unit(c[0], c[1])


def _normal(pos, elem, it, tag, seed):
    c = _philox(pos, elem, it, tag, seed)
    return torch.sqrt(-2.0 * torch.log(_unit(c[0], c[1]))) * torch.cos(2.0 * math.pi * _unit(c[2], c[3]))


def _gamma(shape, it, tag, seed):
    """Gamma(shape, 1) by Marsaglia and Tsang, element e of the flattened
    tensor from substream (e, it, tag)."""
    a = shape.reshape(-1)
    d = torch.where(a < 1.0, a + 1.0, a) - 1.0 / 3.0
    c = 1.0 / torch.sqrt(9.0 * d)
    x = torch.empty_like(a)
    left, pos = torch.arange(a.numel(), device=DEV), 0
    while left.numel():
        z, u = _normal(pos, left, it, tag, seed), _uniform(pos + 1, left, it, tag, seed)
        pos += 2
        V = (1.0 + c[left] * z) ** 3
        ok = V > 0.0
        ok &= torch.log(u) < 0.5 * z * z + d[left] * (1.0 - V + torch.log(torch.where(ok, V, torch.ones_like(V))))
        got = left[ok]
        boost = torch.where(a[got] < 1.0, _uniform(pos, got, it, tag, seed) ** (1.0 / a[got]), torch.ones_like(a[got]))
        x[got] = d[got] * V[ok] * boost
        left = left[~ok]
    return x.reshape(shape.shape)


def _exact_lda(case, seed):
    K, V, D = case["K"], case["V"], case["D"]
    off, w, z = _corpus(case, seed)
    doc = np.repeat(np.arange(D), np.diff(off))
    dk = np.bincount(doc.astype(np.int64) * K + z, minlength=D * K).reshape(D, K)
    kw = np.bincount(z.astype(np.int64) * V + w, minlength=K * V).reshape(K, V)
    gt = _gamma(torch.as_tensor(dk, device=DEV).double() + 0.1, 0, 2, seed)
    gp = _gamma(torch.as_tensor(kw, device=DEV).double() + 0.01, 0, 3, seed)
    phi = torch.zeros((V, (K + 3) // 4 * 4), dtype=torch.float64, device=DEV)
    phi[:, :K] = (gp / gp.sum(1, keepdim=True)).t()
    return {"theta": gt / gt.sum(1, keepdim=True), "phiT": phi, "z": None}


def _mvn_ll(y, m, cov):
    L = torch.linalg.cholesky(cov)
    s = torch.linalg.solve_triangular(L, (y - m).t(), upper=False)
    return -0.5 * y.shape[1] * math.log(2 * math.pi) - torch.log(L.diagonal()).sum() - 0.5 * (s * s).sum(0)


def _exact_mixture(case, seed):
    K, d, move = case["K"], case["d"], case["move"]
    if move == "mwg":
        return None
    Y, z, mu, covs, pis = _mixture(case, seed)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=DEV).double()
    Y, mu, covs, zt = t(Y), t(mu), t(covs), torch.as_tensor(z, device=DEV)
    eye = torch.eye(d, dtype=torch.float64, device=DEV)
    cov0 = 25.0 * eye
    rows = torch.arange(d, device=DEV)
    new_mu, new_cov = torch.empty_like(mu), torch.empty_like(covs)
    for k in range(K):
        yk = Y[zt == k]
        n = yk.shape[0]
        if move == "eslice":
            nu = torch.linalg.cholesky(cov0) @ _normal(rows, k, 0, 10, seed)
            us = iter(_uniform(torch.arange(d, d + 500, device=DEV), k, 0, 10, seed).tolist())
            zero = torch.zeros(d, dtype=torch.float64, device=DEV)
            ll = lambda m: float(_mvn_ll(m[None], zero, cov0)[0] + _mvn_ll(yk, m, covs[k]).sum())
            level = ll(mu[k]) + math.log(next(us))
            ang = next(us) * 2.0 * math.pi
            lo, hi = ang - 2.0 * math.pi, ang
            m = mu[k]
            while hi - lo >= 1e-8:
                cand = mu[k] * math.cos(ang) + nu * math.sin(ang)
                if ll(cand) > level:
                    m = cand
                    break
                lo, hi = (ang, hi) if ang < 0 else (lo, ang)
                ang = lo + next(us) * (hi - lo)
            new_mu[k] = m
            continue
        prec = n * torch.linalg.inv(covs[k])
        post = torch.linalg.inv(torch.linalg.inv(cov0) + prec)
        mean = post @ (prec @ (yk.sum(0) / max(1, n)))
        new_mu[k] = mean + torch.linalg.cholesky(post) @ _normal(rows, k, 0, 8, seed)
        if move == "hier":
            c = yk - new_mu[k]
            S = c.t() @ c + eye
            df = n + d + 2
            A = torch.zeros((d, d), dtype=torch.float64, device=DEV)
            for i in range(d):
                A[i, :i] = _normal(i * df + torch.arange(i, device=DEV), k, 0, 9, seed)
                A[i, i] = torch.sqrt((_normal(i * df + i + torch.arange(df - i, device=DEV), k, 0, 9, seed) ** 2).sum())
            A = torch.linalg.cholesky(torch.linalg.inv(S)) @ A
            new_cov[k] = torch.linalg.inv(A @ A.t())
    out = {"mu": new_mu, "z": None}
    if move == "hier":
        g = _gamma(1.0 + torch.bincount(zt.long(), minlength=K).double(), 0, 7, seed)
        out.update(pis=g / g.sum(), cov=new_cov)
    return out


def _exact_chains(case, seed):
    if case["method"] != "hmc":
        return None
    X, y, init = _regression(case, seed)
    C, D = case["C"], case["D"]
    X = torch.as_tensor(X, device=DEV)
    X = (X.bfloat16() if case["dtype"] == "bf16" else X).double()
    s = 2.0 * torch.as_tensor(y, device=DEV).double() - 1.0
    par = torch.as_tensor(init, device=DEV)[:, [*range(D), D + 1]].clone()
    lsig = torch.nn.functional.logsigmoid

    def density(q):
        th, v = q[:, :D], q[:, D]
        t = th @ X.t()
        sq = (th * th).sum(1)
        good = v > 0.0
        vs = torch.where(good, v, torch.ones_like(v))
        ll = torch.where(good, -2.0 * torch.log(vs) - 1.0 / vs - D * torch.log(vs) - 0.5 * sq / vs,
                         torch.full_like(v, -1e8 * (D + 1))) + lsig(s * t).sum(1)
        g = torch.empty_like(q)
        g[:, :D] = (s * torch.sigmoid(-s * t)) @ X - th / v[:, None]
        g[:, D] = -2.0 / v + 1.0 / (v * v) - 0.5 * D * v + 0.5 * sq / (v * v)
        return ll, g

    c = torch.arange(C, device=DEV)
    stats = torch.zeros((C, 1, 5), dtype=torch.float64, device=DEV)
    P = D + 1
    for it in range(case["iters"]):
        p = _normal(0, c[:, None] * P + torch.arange(P, device=DEV), it, 4, seed)
        u = [_uniform(i, c, it, 5, seed) for i in range(3)]
        eps = (0.8 + 0.4 * u[0]) * 0.01
        L = torch.clamp(torch.round((0.9 + 0.2 * u[1]) * 0.1 / eps), min=1.0)
        ll0, g = density(par)
        k0 = 0.5 * (p * p).sum(1)
        e = eps[:, None]
        q, p = par, p + 0.5 * e * g
        ll1, q1, p1 = ll0.clone(), q.clone(), p.clone()
        for step in range(1, int(L.max()) + 1):
            q = q + e * p
            ll, g = density(q)
            end = L == step
            ll1[end], q1[end], p1[end] = ll[end], q[end], (p + 0.5 * e * g)[end]
            p = p + e * g
        gain = ll1 - ll0 + k0 - 0.5 * (p1 * p1).sum(1)
        ok = torch.log(u[2]) < gain
        par = torch.where(ok[:, None], q1, par)
        stats[:, 0, 0] += ok.double()
        stats[:, 0, 4] += (~(gain > -1000.0)).double()
    full = torch.as_tensor(init, device=DEV).clone()
    full[:, :D], full[:, D + 1] = par[:, :D], par[:, D]
    return {"pars": full, "stats": stats}


def _exact_logistic(X, y, theta, want_logp, want_grad):
    """Data part of log density and gradient, rows in slices."""
    th = theta.double()
    C, D = th.shape
    logp = torch.zeros(C, dtype=torch.float64, device=DEV)
    grad = torch.zeros((C, D), dtype=torch.float64, device=DEV)
    step = max(1024, (1 << 26) // max(C, D))
    for a in range(0, X.shape[0], step):
        x, s = X[a:a + step].double(), 2.0 * y[a:a + step].double() - 1.0
        t = s[:, None] * (x @ th.t())
        if want_logp:
            logp += torch.nn.functional.logsigmoid(t).sum(0)
        if want_grad:
            grad += (s[:, None] * torch.sigmoid(-t)).t() @ x
    return th, logp, grad


def _exact_pass(case, seed):
    X, y, theta = _pass_inputs(case, seed)
    th, logp, grad = _exact_logistic(X, y, theta, case["mode"] != "grad", case["mode"] != "logp")
    logp += (math.lgamma(2.0) - math.lgamma(1.5) - 0.5 * math.log(3.0 * math.pi) - 2.0 * torch.log1p(th * th / 3.0)).sum(1)
    grad -= 4.0 * th / (3.0 + th * th)
    return {"logp": logp if case["mode"] != "grad" else None, "grad": grad if case["mode"] != "logp" else None}


def _exact_group(case, seed):
    logps, grads = [], []
    for X, y, theta in _group_inputs(case, seed):
        th, logp, grad = _exact_logistic(X, y, theta, True, True)
        logps.append(logp - (0.5 * math.log(2.0 * math.pi) + 0.5 * th * th).sum(1))
        grads.append((grad - th).view(-1))
    return {"logp": torch.cat(logps), "grad": torch.cat(grads)}


def _layers(D, h, seed):
    """The network's initial weights: Glorot-uniform from the seed, zero
    biases, the last layer's weights scaled by 0.1."""
    rs = np.random.default_rng(seed)
    out = []
    for i, (fi, fo) in enumerate(((D, h), (h, h), (h, D))):
        lim = math.sqrt(6.0 / (fi + fo))
        w = rs.uniform(-lim, lim, fi * fo).astype(np.float32)
        w = w * np.float32(0.1) if i == 2 else w
        out += [torch.as_tensor(w, device=DEV).double().view(fo, fi), torch.zeros(fo, dtype=torch.float64, device=DEV)]
    return out


def _exact_surrogate(case, seed):
    D, h = case["D"], 256
    buf, grad, at = _pairs(case, seed)
    buf, grad, at = buf.double(), grad.double(), at.double()
    mu, a = buf.mean(0), grad.mean(0)
    dt = buf - mu
    inv_s = (dt * dt).mean(0).rsqrt()
    A = dt.t() @ dt
    M = torch.linalg.solve(A + torch.eye(D, dtype=torch.float64, device=DEV) * (1e-9 * A.diagonal().mean()),
                           dt.t() @ (grad - a))
    res = grad - a - dt @ M
    o = (res * res).mean(0).sqrt()
    W = _layers(D, h, seed)
    low = lambda w: w.bfloat16().double()
    gelu = torch.nn.functional.gelu

    def forward(z, W):
        p1 = z @ low(W[0]).t() + W[1]
        p2 = gelu(p1) @ low(W[2]).t() + W[3]
        return p1, p2, gelu(p2) @ low(W[4]).t() + W[5]

    if case["mode"] == "predict":
        d = at - mu
        return {"grad": a + d @ M + o * forward(d * inv_s, W)[2]}
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) + 1)
    B, steps = 512, case["steps"]
    idx = torch.randint(0, BUFFER, (steps * B,), generator=gen, device=DEV)
    zs, ts = dt[idx] * inv_s, res[idx] / o
    m, v = [torch.zeros_like(w) for w in W], [torch.zeros_like(w) for w in W]

    def dgelu(x):
        return 0.5 * (1.0 + torch.erf(x * math.sqrt(0.5))) + x * torch.exp(-0.5 * x * x) / math.sqrt(2.0 * math.pi)

    for i in range(steps):
        z, t = zs[i * B:(i + 1) * B], ts[i * B:(i + 1) * B]
        p1, p2, y = forward(z, W)
        loss = ((y - t) ** 2).sum() / (B * D)
        dy = 2.0 * (y - t) / (B * D)
        d2 = (dy @ low(W[4])) * dgelu(p2)
        d1 = (d2 @ low(W[2])) * dgelu(p1)
        gs = [d1.t() @ z, d1.sum(0), d2.t() @ gelu(p1), d2.sum(0), dy.t() @ gelu(p2), dy.sum(0)]
        for j, g in enumerate(gs):
            m[j] = 0.9 * m[j] + 0.1 * g
            v[j] = 0.999 * v[j] + 0.001 * g * g
            W[j] = W[j] - 1e-3 * (m[j] / (1.0 - 0.9 ** (i + 1))) / ((v[j] / (1.0 - 0.999 ** (i + 1))).sqrt() + 1e-8)
    flat = lambda q: torch.cat([x.reshape(-1) for x in q])
    return {"loss": loss, "w": flat(W), "m": flat(m), "v": flat(v)}


def exact(case, seed):
    return {"lda": _exact_lda, "mixture": _exact_mixture, "chains": _exact_chains, "pass": _exact_pass,
            "group": _exact_group, "surrogate": _exact_surrogate}[case["kind"]](case, seed)
