"""The calls this engine's users make, as timed cases.

Each case is one pass through a public entry point of the `riskgpu` binding, with seeded synthetic inputs of the
shapes that `riskgpu/synth.py` and the benchmark use.  Kinds:

  plugin    the reference's plugin call, get_cuda_model().run_model, from host (GSL layout) mu and Sigma
  oneshot   rg_run: host mu, Sigma and weights in, estimates out; the factor is built and dropped in the call
  simulate  rg_simulate on a resident portfolio (FP32 or tensor-core form, daily or aggregated draws, VaR/CVaR,
            per-path outputs)
  batch     many portfolios of uneven size in one rg_batch launch
  returns   a daily-returns matrix to mu, Sigma, the realised crash frequency and a resident FP64 factor

`exact` restates the model in 64 bits with plain torch: Philox4x32-10 words (key = seed, counter = (block, 0, path)),
Box-Muller, R = H mu + L Zsum with L L^T = Sigma.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "gpu-montecarlo-risk_gb300"))

import riskgpu  # noqa: E402
from riskgpu import synth  # noqa: E402

PRECISION = {"auto": riskgpu.PREC_AUTO, "bf16x3": riskgpu.PREC_BF16X3, "fp16x3": riskgpu.PREC_FP16X3}


def listed():
    return [
        # the reference's published setting (9 indices, x = 2 %, k = 5) at its configuration's default path count:
        # the smallest call a switching user makes
        dict(name="plugin_9", kind="plugin", n=9, paths=100_000),
        # the same call drawing the reference kernel's own XORWOW stream, for results equal to the reference's
        dict(name="xorwow_9", kind="simulate", n=9, paths=1_000_000, horizon=1, precision="auto", draws="daily",
             var=False, per_path=False, rng="xorwow"),
        # the drop-in benchmark workload: 50 one-factor assets, 1e8 one-day paths
        dict(name="plugin_50", kind="plugin", n=50, paths=100_000_000),
        # the small risk report: 20 assets, 1e6 paths, 99 % VaR and CVaR
        dict(name="var_20", kind="simulate", n=20, paths=1_000_000, horizon=1, precision="auto", draws="daily",
             var=True, per_path=False, rng="philox"),
        # S and w.R of every path kept for a later analysis; ragged assets and paths, ten summed days
        dict(name="paths_61", kind="simulate", n=61, paths=200_003, horizon=10, precision="auto", draws="daily",
             var=False, per_path=True, rng="philox"),
        # the plain FP32 form of the large benchmark portfolio
        dict(name="fp32_600", kind="simulate", n=600, paths=500_000, horizon=10, precision="auto", draws="daily",
             var=False, per_path=False, rng="philox"),
        # the benchmark's headline: 600 assets, ten summed days, BF16 hi+lo on the tensor cores, with VaR/CVaR
        dict(name="bf16_600", kind="simulate", n=600, paths=4_000_000, horizon=10, precision="bf16x3",
             draws="daily", var=True, per_path=False, rng="philox"),
        # the FP16 split with one N(0, H) draw an asset: the form for long horizons; ragged assets and paths
        dict(name="fp16_487", kind="simulate", n=487, paths=2_000_001, horizon=20, precision="fp16x3",
             draws="aggregated", var=False, per_path=False, rng="philox"),
        # an interactive what-if on a resident portfolio: few paths, the answer's latency is what counts
        dict(name="whatif_333", kind="simulate", n=333, paths=5_000, horizon=5, precision="bf16x3", draws="daily",
             var=False, per_path=False, rng="philox"),
        # end to end from host arrays, as a program with a new covariance each call does it
        dict(name="oneshot_600", kind="oneshot", n=600, paths=100_000, horizon=10, precision="bf16x3",
             draws="daily", var=False, per_path=False, rng="philox"),
        # uneven portfolios (10..600 assets, 1..20 days, 1e4..1e6 paths) in one launch
        dict(name="batch_24", kind="batch", count=24, n_max=600, m_min=10_000, m_max=1_000_000),
        # 2000 days of 600 returns to a resident factor, with the realised crash frequency
        dict(name="returns_600", kind="returns", n=600, days=2000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _most_paths(n, horizon):
    # as much work as the largest listed case does: 2.4e10 normals of a 600-asset contraction
    return max(1000, int(1.2e10 / (n * (horizon + n / 60.0))))


def draw(rng):
    kind = rng.choice(["plugin", "simulate", "simulate", "tensor", "tensor", "oneshot", "batch", "returns", "xorwow"])
    if kind == "plugin":
        n = _log(rng, 2, 64)
        return dict(kind="plugin", n=n, paths=_log(rng, 10_000, min(100_000_000, _most_paths(n, 1))))
    if kind == "xorwow":
        n = _log(rng, 2, 64)
        return dict(kind="simulate", n=n, paths=_log(rng, 10_000, 1_000_000), horizon=1, precision="auto",
                    draws="daily", var=False, per_path=rng.random() < 0.5, rng="xorwow")
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(2, 24), n_max=rng.choice([60, 200, 400, 600]), m_min=1_000,
                    m_max=_log(rng, 20_000, 500_000))
    if kind == "returns":
        n = _log(rng, 5, 700)
        return dict(kind="returns", n=n, days=n + _log(rng, 250, 2000))
    tensor = kind != "simulate" and (kind == "tensor" or rng.random() < 0.5)
    n = _log(rng, 65, 640) if tensor else _log(rng, 2, 768)
    horizon = rng.choice([1, 1, 2, 5, 10, 20])
    case = dict(kind="oneshot" if kind == "oneshot" else "simulate", n=n,
                paths=_log(rng, 1_000, min(20_000_000, _most_paths(n, horizon))), horizon=horizon,
                precision=rng.choice(["bf16x3", "fp16x3"]) if tensor else "auto",
                draws=rng.choice(["daily", "daily", "aggregated"]), var=rng.random() < 0.4, per_path=False,
                rng="philox")
    if case["kind"] == "simulate":
        case["per_path"] = rng.random() < 0.3
    return case


# ------------------------------------------------------------------------------------------------ inputs
def _inputs(n, horizon, seed, factors):
    """mu, Sigma, weights, thresholds and the path seed of one portfolio."""
    rng = np.random.default_rng(seed)
    if factors == 1:
        mu, sigma, _, _ = synth.one_factor_sigma(rng, n)
        x, k = 0.02 * math.sqrt(horizon), 5 if n == 9 else max(1, n // 4)
    else:
        mu, sigma, _, _ = synth.factor_sigma(rng, n, factors, 0.005)
        x, k = 0.028 * math.sqrt(horizon), max(1, n // 10)
    w = rng.dirichlet(np.ones(n))
    sd = math.sqrt(horizon * float(w @ sigma @ w))
    thr = horizon * float(w @ mu) - 1.645 * sd  # about the 5 % quantile
    return dict(mu=mu, sigma=sigma, w=w, x=x, k=k, thr=thr, seed=int(rng.integers(1, 2 ** 31)), horizon=horizon)


def _factors(case):
    return 1 if case["kind"] == "plugin" or case["n"] <= 64 else 5


def _batch_inputs(case, seed):
    rng = np.random.default_rng(seed)
    items = []
    for _ in range(case["count"]):
        n, h = int(rng.integers(10, case["n_max"] + 1)), int(rng.integers(1, 21))
        m = int(round(math.exp(rng.uniform(math.log(case["m_min"]), math.log(case["m_max"])))))
        items.append(dict(_inputs(n, h, int(rng.integers(1, 2 ** 31)), 3), paths=m))
    return items


def _returns_inputs(case, seed):
    rng = np.random.default_rng(seed)
    mu, _, B, idio = synth.factor_sigma(rng, case["n"], 5, 0.005)
    X = mu + rng.normal(size=(case["days"], 5)) @ B.T + rng.normal(size=(case["days"], case["n"])) * idio
    return np.ascontiguousarray(X)


def _query(case, p, **more):
    return riskgpu.make_query(
        case.get("paths", p.get("paths")), p["seed"], x=p["x"], k=p["k"], horizon=p["horizon"],
        port_threshold=p["thr"], rng=riskgpu.RNG_XORWOW_REF if case.get("rng") == "xorwow" else riskgpu.RNG_PHILOX,
        precision=PRECISION[case.get("precision", "auto")], var_level=0.99 if case.get("var") else 0.0,
        draw_mode=riskgpu.DRAWS_AGGREGATED if case.get("draws") == "aggregated" else riskgpu.DRAWS_DAILY, **more)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "plugin":
        p = _inputs(case["n"], 1, seed, _factors(case))
        return dict(case=case, p=p, call=riskgpu.PluginCall(p["mu"], p["sigma"]))
    if kind == "batch":
        items = _batch_inputs(case, seed)
        pairs = []
        for p in items:
            q = riskgpu.make_query(p["paths"], p["seed"], x=p["x"], k=p["k"], horizon=p["horizon"],
                                   port_threshold=p["thr"], precision=riskgpu.PREC_BF16X3)
            pairs.append((riskgpu.Portfolio(p["mu"], p["sigma"], p["w"]), q))
        return dict(case=case, batch=riskgpu.Batch(pairs))
    if kind == "returns":
        return dict(case=case, returns=_returns_inputs(case, seed))
    p = _inputs(case["n"], case["horizon"], seed, _factors(case))
    if kind == "oneshot":
        return dict(case=case, p=p, query=_query(case, p))
    state = dict(case=case, port=riskgpu.Portfolio(p["mu"], p["sigma"], p["w"]))
    more = {}
    if case["per_path"]:
        state["S"] = torch.zeros(case["paths"], dtype=torch.int32, device="cuda")
        state["W"] = torch.zeros(case["paths"], dtype=torch.float32, device="cuda")
        more = dict(d_s_values=state["S"].data_ptr(), d_port_values=state["W"].data_ptr())
    state["query"] = _query(case, p, **more)
    return state


# ------------------------------------------------------------------------------------------------ one pass
ESTIMATES = ("crash_count", "breach_count", "p_crash", "se_crash", "ci_lower", "ci_upper", "p_breach", "se_breach")


def _estimates(r, var):
    out = {f: r[f] for f in ESTIMATES}
    if var:
        out.update(var=r["var"], cvar=r["cvar"], tail_count=r["tail_count"])
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "plugin":
        p = state["p"]
        r = state["call"].run(case["paths"], p["k"], p["x"], p["seed"])
        return {f: r[f] for f in ("status", "count", "P_hat", "std_error", "ci_lower", "ci_upper")}
    if kind == "batch":
        return [[r["crash_count"], r["breach_count"]] for r in state["batch"].run()]
    if kind == "returns":
        X = state["returns"]
        mu, sigma = riskgpu.moments(X)
        freq = riskgpu.crash_frequency(X, 0.02, max(1, X.shape[1] // 4))
        port = riskgpu.Portfolio(mu, sigma, np.full(X.shape[1], 1.0 / X.shape[1]))
        info = port.info()
        L = port.factor()
        port.close()
        return dict(mu=mu, sigma=sigma, frequency=freq, factor=L, variance=info["wsw"], mean=info["wmu"])
    if kind == "oneshot":
        p = state["p"]
        return _estimates(riskgpu.run(p["mu"], p["sigma"], p["w"], state["query"]), case["var"])
    out = _estimates(state["port"].simulate(state["query"]), case["var"])
    if case["per_path"]:
        out.update(S=state["S"], port=state["W"])
    return out


# ------------------------------------------------------------------------------------------------ work
def _mc_work(n, horizon, paths, draws):
    # a drawn normal: 10 integer multiplies and xors of Philox and 6 operations of Box-Muller; the contraction is
    # a triangle; then the compare and the weighted sum
    normals = n * (1 if draws == "aggregated" else horizon)
    return paths * (16.0 * normals + n * (n + 1.0) + 3.0 * n)


def work(case):
    kind = case["kind"]
    if kind == "returns":
        n, t = case["n"], case["days"]
        return {"bytes": 8.0 * (t * n + 2 * n * n + n), "flops": t * n * (n + 1.0) + n ** 3 / 3.0 + 2.0 * t * n}
    if kind == "batch":
        m = (case["m_max"] - case["m_min"]) / math.log(case["m_max"] / case["m_min"])  # means of the distributions
        n = 0.5 * (10 + case["n_max"])
        return {"bytes": case["count"] * 8.0 * n * n, "flops": case["count"] * _mc_work(n, 10.5, m, "daily")}
    n, paths = case["n"], case["paths"]
    out = 8.0 * paths if case.get("per_path") else 0.0
    return {"bytes": 8.0 * n * (n + 1) + 36 + out,
            "flops": _mc_work(n, case.get("horizon", 1), paths, case.get("draws", "daily"))}


# ------------------------------------------------------------------------------------------------ 64 bits
def _mulhilo(m, v):
    p = v * m  # the low 64 bits are right, also where the sign bit is set
    return (p >> 32) & 0xFFFFFFFF, p & 0xFFFFFFFF


def _philox(block, path, seed):
    c0, c1, c2, c3 = block, torch.zeros_like(block), path & 0xFFFFFFFF, (path >> 32) & 0xFFFFFFFF
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        h0, l0 = _mulhilo(0xD2511F53, c0)
        h1, l1 = _mulhilo(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def _pair(a, b):
    u = 1.0 - (a >> 9).double() * 2.0 ** -23
    t = (2.0 * math.pi) * ((b >> 9).double() * 2.0 ** -23)
    r = torch.sqrt(-2.0 * torch.log(u))
    return r * torch.cos(t), r * torch.sin(t)


def _simulate64(p, paths, aggregated, per_path, var, weights=True):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n, h = p["mu"].shape[0], p["horizon"]
    nq = (n + 3) // 4
    L = torch.linalg.cholesky(torch.from_numpy(p["sigma"])).to(dev)
    mu, w = (h * torch.from_numpy(p["mu"])).to(dev), torch.from_numpy(p["w"]).to(dev)
    days, scale = (1, math.sqrt(h)) if aggregated else (h, 1.0)
    crash = breach = 0
    S_all, W_all = [], []
    step = max(1, 8_000_000 // nq)
    for p0 in range(0, paths, step):
        path = torch.arange(p0, min(paths, p0 + step), dtype=torch.int64, device=dev)[:, None]
        z = torch.zeros(path.shape[0], nq, 4, dtype=torch.float64, device=dev)
        for d in range(days):
            block = (d * nq + torch.arange(nq, dtype=torch.int64, device=dev))[None, :].expand(path.shape[0], nq)
            a, b, c, e = _philox(block, path.expand(-1, nq), p["seed"])
            z[:, :, 0:2] += torch.stack(_pair(a, b), 2)
            z[:, :, 2:4] += torch.stack(_pair(c, e), 2)
        R = mu + scale * (z.reshape(path.shape[0], 4 * nq)[:, :n] @ L.T)
        S, W = (R < -p["x"]).sum(1), R @ w
        crash += int((S >= p["k"]).sum())
        breach += int((W < p["thr"]).sum()) if weights else 0
        if per_path:
            S_all.append(S.to(torch.int32))
        if per_path or var:
            W_all.append(W)
    return crash, breach, torch.cat(S_all) if per_path else None, torch.cat(W_all) if per_path or var else None


def _normals(p, paths, aggregated):
    return float(paths) * p["mu"].shape[0] * (1 if aggregated else p["horizon"])


def _stats(count, m):
    P = count / m
    se = math.sqrt(P * (1.0 - P) / m)
    return P, se, max(0.0, P - 1.96 * se), min(1.0, P + 1.96 * se)


def exact(case, seed):
    kind = case["kind"]
    if kind == "returns":
        X = _returns_inputs(case, seed)
        n = X.shape[1]
        mu = X.mean(0)
        D = X - mu
        sigma = D.T @ D / (X.shape[0] - 1)
        w = np.full(n, 1.0 / n)
        return dict(mu=mu, sigma=sigma, frequency=float(((X < -0.02).sum(1) >= max(1, n // 4)).mean()),
                    factor=np.linalg.cholesky(sigma), variance=float(w @ sigma @ w), mean=float(w @ mu))
    if kind == "batch":
        return None  # whole numbers only
    if case.get("rng") == "xorwow":
        return None  # the stream is cuRAND's
    aggregated = case.get("draws") == "aggregated"
    p = _inputs(case["n"], case.get("horizon", 1), seed, _factors(case))
    if _normals(p, case["paths"], aggregated) > 2.6e10:
        return None
    var, per_path = bool(case.get("var")), bool(case.get("per_path"))
    m = case["paths"]
    crash, breach, S, W = _simulate64(p, m, aggregated, per_path, var, weights=kind != "plugin")
    P, se, lo, hi = _stats(crash, m)
    if kind == "plugin":
        return dict(status=None, count=None, P_hat=P, std_error=se, ci_lower=lo, ci_upper=hi)
    Pb, seb, _, _ = _stats(breach, m)
    out = dict(crash_count=None, breach_count=None, p_crash=P, se_crash=se, ci_lower=lo, ci_upper=hi, p_breach=Pb,
               se_breach=seb)
    if var:
        T = min(m, max(1, math.ceil(0.01 * m - 1e-9)))
        tail = torch.topk(W, T, largest=False).values
        out.update(var=float(-tail[-1]), cvar=float(-tail.mean()), tail_count=None)
    if per_path:
        out.update(S=None, port=W)
    return out
