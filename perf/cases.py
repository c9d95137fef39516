"""Performance cases of the pricing engine: what its users have it do, through its public entry points.

`listed()` names one case for each kind of call, `draw(rng)` gives another one of the same ranges.  A case is a dict of
plain values: the kind of call, its sizes and its options.  The contract terms and the market come from the seed
(`prepare`); `run` makes the call; `work` states what the call cannot do without; `exact` evaluates the same draws in
64 bits with plain torch.

Prices of the engine's FP64 mode come back as float64 arrays, those of its FP32 mode as float32 arrays.
"""
import math
import random

import numpy as np
import torch

import openferric_b200 as of
from openferric_b200.adjoint import HestonAdjointSpec, heston_adjoint
from openferric_b200.book import BookEntry, price_book, price_book_greeks
from openferric_b200.gpu_mc import mc_european_gpu
from openferric_b200.lsm import LongstaffSchwartzEngine

_VR = {"none": of.VarianceReduction.None_, "antithetic": of.VarianceReduction.Antithetic}


def listed():
    return [
        # One European through the pricing engine as it comes (FP64, the reference's streams): 100,000 paths of daily
        # steps over a year, the benchmark of the reference's pricing engine.
        {"name": "european", "kind": "european", "paths": 100_000, "steps": 252, "vr": "none"},
        # A daily-fixing arithmetic Asian with the geometric control variate, as the Asian engine prices it
        # (FP64, antithetic pairs).
        {"name": "asian", "kind": "asian", "paths": 100_000, "steps": 252, "fixings": 252, "cv": True},
        # A discretely monitored knock-out with antithetic pairs (FP64); 20 trading days x 6 and an odd path count.
        {"name": "barrier", "kind": "barrier", "paths": 50_001, "steps": 126, "style": "up_out", "vr": "antithetic"},
        # A European under Heston (FP64, full-truncation Euler), the path-generator interface.
        {"name": "heston", "kind": "heston", "paths": 131_072, "steps": 256, "vr": "none"},
        # A European with its pathwise Greeks (FP64), what a risk report asks of the pricing engine.
        {"name": "greeks", "kind": "greeks", "paths": 120_000, "steps": 64, "vr": "antithetic"},
        # An American put by least squares (FP64, the reference's stream), the Longstaff-Schwartz table's settings.
        {"name": "american", "kind": "american", "paths": 100_000, "steps": 50},
        # A book of American puts with deltas (FP32, cubic basis), one call: the largest case.
        {"name": "american_batch", "kind": "american_batch", "contracts": 64, "paths": 1 << 20, "steps": 50},
        # A strike strip under Heston on one path set (FP32): a smile, 41 strikes, 2^20 paths of 256 steps.
        {"name": "strip", "kind": "strip", "model": "heston", "paths": 1 << 20, "steps": 256, "strikes": 41,
         "vr": "none"},
        # The smallest call: one European on the FP32 path kernel, a few thousand short paths, where latency counts.
        {"name": "quick", "kind": "quick", "paths": 10_000, "steps": 16},
        # A mixed book (European, daily Asian, up-and-out) of some hundred options with their own paths and daily
        # steps, in one call (FP32).
        {"name": "book", "kind": "book", "options": 384, "log2_min": 14, "log2_max": 17, "vr": "none"},
        # The same kind of book with delta, vega, rho and theta of every option (FP32, pathwise), a smaller one.
        {"name": "book_greeks", "kind": "book_greeks", "options": 192, "log2_min": 13, "log2_max": 15,
         "vr": "antithetic"},
        # A daily-fixing Asian under Heston QE with all seven sensitivities from the adjoint (FP32).
        {"name": "adjoint", "kind": "adjoint", "paths": 1 << 20, "steps": 512, "asian": True},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["european", "asian", "barrier", "heston", "greeks", "american", "american_batch", "strip",
                       "quick", "book", "book_greeks", "adjoint"])
    vr = rng.choice(["none", "antithetic"])
    if kind in ("european", "greeks"):
        return {"kind": kind, "paths": log(2_000, 400_000), "steps": log(2, 365), "vr": vr}
    if kind == "asian":
        steps = log(12, 365)
        return {"kind": kind, "paths": log(2_000, 200_000), "steps": steps,
                "fixings": rng.choice([steps, max(2, steps // 5), 12]), "cv": rng.random() < 0.7}
    if kind == "barrier":
        return {"kind": kind, "paths": log(2_000, 200_000), "steps": log(12, 365),
                "style": rng.choice(["up_out", "up_in", "down_out", "down_in"]), "vr": vr}
    if kind == "heston":
        return {"kind": kind, "paths": log(4_000, 262_144), "steps": log(16, 256), "vr": vr}
    if kind == "american":
        return {"kind": kind, "paths": log(10_000, 200_000), "steps": log(10, 100)}
    if kind == "american_batch":
        return {"kind": kind, "contracts": log(2, 64), "paths": log(1 << 16, 1 << 19), "steps": log(25, 100)}
    if kind == "strip":
        return {"kind": kind, "model": rng.choice(["gbm", "heston", "qe"]), "paths": log(1 << 14, 1 << 20),
                "steps": log(8, 256), "strikes": log(1, 64), "vr": vr}
    if kind == "quick":
        return {"kind": kind, "paths": log(4_000, 1 << 20), "steps": log(1, 252)}
    if kind == "book":
        return {"kind": kind, "options": log(12, 384), "log2_min": 12, "log2_max": rng.choice([14, 16]), "vr": vr}
    if kind == "book_greeks":
        return {"kind": kind, "options": log(12, 192), "log2_min": 12, "log2_max": rng.choice([13, 15]), "vr": vr}
    return {"kind": "adjoint", "paths": log(1 << 15, 1 << 20), "steps": log(16, 512), "asian": rng.random() < 0.5}


# ---- the terms of a case, from its seed -----------------------------------


def _terms(case, seed):
    """Market, contract and stream of a single-option case."""
    g = random.Random(seed * 1_000_003 + 17)
    t = {"spot": g.uniform(80.0, 120.0), "rate": g.uniform(0.01, 0.06), "vol": g.uniform(0.15, 0.45),
         "expiry": g.uniform(0.5, 2.0), "seed": g.randrange(1 << 31)}
    t["strike"] = t["spot"] * g.uniform(0.9, 1.1)
    t["call"] = g.random() < 0.5
    t["level"] = t["spot"] * (g.uniform(1.15, 1.4) if case.get("style", "up").startswith("up") else g.uniform(0.7, 0.9))
    t.update(kappa=g.uniform(1.0, 3.0), theta=g.uniform(0.03, 0.08), xi=g.uniform(0.3, 0.6), rho=g.uniform(-0.8, -0.4),
             v0=g.uniform(0.03, 0.08))
    return t


def _fixing_times(case, t):
    n = case["fixings"]
    return [t["expiry"] * (j / n) for j in range(1, n + 1)]


def _strikes(case, t):
    n = case["strikes"]
    return [t["spot"] * (0.8 + 0.4 * (k + 0.5) / n) for k in range(n)]


def _puts(case, seed):
    """Spots and vols of a batch of American puts at strike 40, rate 6 %, 50 exercise dates a year."""
    g = np.random.default_rng(seed + 5)
    n = case["contracts"]
    return g.uniform(30.0, 50.0, n), g.choice([0.2, 0.4], n), int(g.integers(1 << 31))


def _book(case, seed):
    g = np.random.default_rng(seed + 9)
    entries = []
    for i in range(case["options"]):
        s0, t = g.uniform(50.0, 150.0), g.uniform(0.1, 5.0)
        steps = max(1, int(round(252 * t)))
        paths = int(round(2.0 ** g.uniform(case["log2_min"], case["log2_max"])))
        entries.append({"s0": s0, "strike": s0 * g.uniform(0.8, 1.2), "vol": g.uniform(0.1, 0.6),
                        "rate": g.uniform(0.0, 0.06), "expiry": t, "steps": steps, "paths": paths,
                        "kind": ("european", "asian", "barrier")[i % 3], "level": s0 * g.uniform(1.1, 1.5)})
    return entries, int(g.integers(1 << 31))


def _market(spot, rate, vol):
    return of.Market.builder().spot(spot).rate(rate).flat_vol(vol).build()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "american_batch":
        spots, vols, stream = _puts(case, seed)
        eng = LongstaffSchwartzEngine(case["paths"], case["steps"], stream) \
            .with_precision(of.Precision.Fp32Philox).with_basis_degree(3)
        put = of.VanillaOption.american_put(40.0, case["steps"] / 50.0)
        return {"kind": kind, "engine": eng, "items": [(put, _market(s, 0.06, v)) for s, v in zip(spots, vols)]}
    if kind in ("book", "book_greeks"):
        entries, stream = _book(case, seed)
        book = []
        for e in entries:
            if e["kind"] == "european":
                inst = of.VanillaOption.european_call(e["strike"], e["expiry"])
            elif e["kind"] == "asian":
                n, T = e["steps"], e["expiry"]
                obs = [T * (j / n) for j in range(1, n + 1)]
                inst = of.AsianOption(of.OptionType.Call, e["strike"], T,
                                      of.AsianSpec(of.Averaging.Arithmetic, of.StrikeType.Fixed, obs))
            else:
                inst = of.BarrierOption(of.OptionType.Call, e["strike"], e["expiry"],
                                        of.BarrierSpec(of.BarrierDirection.Up, of.BarrierStyle.Out, e["level"], 0.0))
            book.append(BookEntry(inst, _market(e["s0"], e["rate"], e["vol"]), e["paths"], e["steps"],
                                  _VR[case["vr"]]))
        return {"kind": kind, "book": book, "seed": stream}
    t = _terms(case, seed)
    opt = of.OptionType.Call if t["call"] else of.OptionType.Put
    df = math.exp(-t["rate"] * t["expiry"])
    state = {"kind": kind, "terms": t, "df": df, "market": _market(t["spot"], t["rate"], t["vol"]),
             "option": of.VanillaOption(opt, t["strike"], t["expiry"])}
    if kind in ("european", "greeks", "barrier"):
        state["engine"] = of.MonteCarloPricingEngine(case["paths"], case["steps"], t["seed"]) \
            .with_variance_reduction(_VR[case["vr"]])
    if kind == "barrier":
        up, out = case["style"].split("_")[0] == "up", case["style"].split("_")[1] == "out"
        state["option"] = of.BarrierOption(
            opt, t["strike"], t["expiry"],
            of.BarrierSpec(of.BarrierDirection.Up if up else of.BarrierDirection.Down,
                           of.BarrierStyle.Out if out else of.BarrierStyle.In, t["level"], 0.0))
    elif kind == "asian":
        state["engine"] = of.ArithmeticAsianMC(case["paths"], case["steps"], t["seed"]) \
            .with_control_variate(case["cv"])
        state["option"] = of.AsianOption(opt, t["strike"], t["expiry"],
                                         of.AsianSpec(of.Averaging.Arithmetic, of.StrikeType.Fixed,
                                                      _fixing_times(case, t)))
    elif kind == "american":
        state["engine"] = LongstaffSchwartzEngine(case["paths"], case["steps"], t["seed"])
        state["option"] = of.VanillaOption.american_put(t["strike"], t["expiry"])
    elif kind in ("heston", "strip"):
        model = of.Heston(t["rate"], t["kappa"], t["theta"], t["xi"], t["rho"], t["v0"])
        if case.get("model") == "gbm":
            state["generator"] = of.GbmPathGenerator(of.Gbm(t["rate"], t["vol"]), t["spot"], t["expiry"], case["steps"])
        else:
            state["generator"] = of.HestonPathGenerator(model, t["spot"], t["expiry"], case["steps"],
                                                        "qe" if case.get("model") == "qe" else "euler")
        state.update(opt=opt, paths=case["paths"], antithetic=case["vr"] == "antithetic")
        if kind == "heston":
            state["engine"] = of.MonteCarloEngine(case["paths"], t["seed"]).with_antithetic(state["antithetic"])
        else:
            state["strikes"] = _strikes(case, t)
    elif kind == "quick":
        state.update(paths=case["paths"], steps=case["steps"])
    elif kind == "adjoint":
        state["spec"] = HestonAdjointSpec(t["strike"], t["expiry"], case["paths"], case["steps"], t["seed"], opt,
                                          case["asian"])
        state["model"] = (t["spot"], t["rate"], t["v0"], t["kappa"], t["theta"], t["xi"], t["rho"])
    return state


def run(state):
    kind = state["kind"]
    if kind in ("european", "asian", "barrier", "american"):
        r = state["engine"].price(state["option"], state["market"])
        return {"price": np.array([r.price]), "stderr": np.array([r.stderr])}
    if kind == "heston":
        p, s = state["engine"].run(state["generator"], state["option"], state["df"])
        return {"price": np.array([p]), "stderr": np.array([s])}
    if kind == "greeks":
        r = state["engine"].price_with_greeks_aad(state["option"], state["market"])
        g = r.greeks
        return {"price": np.array([r.price]), "stderr": np.array([r.stderr]),
                "greeks": np.array([g.delta, g.vega, g.theta, g.rho])}
    if kind == "american_batch":
        rs = state["engine"].price_batch(state["items"], with_delta=True)
        return {"price": _f32(r.price for r in rs), "stderr": _f32(r.stderr for r in rs),
                "delta": _f32(r.greeks.delta for r in rs)}
    if kind == "strip":
        rs = of.price_strike_strip(state["generator"], state["opt"], state["strikes"], state["paths"],
                                   state["terms"]["seed"], state["df"], antithetic=state["antithetic"])
        return {"price": _f32(p for p, _ in rs), "stderr": _f32(s for _, s in rs)}
    if kind == "quick":
        t = state["terms"]
        r = mc_european_gpu(t["spot"], t["strike"], t["rate"], t["vol"], t["expiry"], state["paths"], state["steps"],
                            t["seed"], t["call"])
        return {"price": _f32([r.price]), "stderr": _f32([r.stderr])}
    if kind == "book":
        rs = price_book(state["book"], state["seed"])
        return {"price": _f32(r.price for r in rs), "stderr": _f32(r.stderr for r in rs)}
    if kind == "book_greeks":
        rs = price_book_greeks(state["book"], state["seed"])
        out = {"price": _f32(r.result.price for r in rs), "stderr": _f32(r.result.stderr for r in rs)}
        for g in ("delta", "vega", "rho", "theta"):
            out[g] = _f32(getattr(r.result.greeks, g) for r in rs)
            out[g + "_se"] = _f32(getattr(r.greeks_stderr, g) for r in rs)
        return out
    r = heston_adjoint(state["spec"], *state["model"])
    return {"price": _f32([r.price]), "stderr": _f32([r.stderr]), "greeks": _f32(r.greeks.values()),
            "greeks_se": _f32(r.greeks_stderr.values())}


def _f32(values):
    return np.array(list(values), dtype=np.float32)


def work(case):
    """Inputs and outputs are a few numbers a contract, except that least squares reads and rewrites its paths and cash
    flows at each date (a store, a reload and the cash flow's read and write).  The flops of a path-step are those of
    its normal and its update with each fma as two and each elementary function as one: 22 for the inverse normal of
    the FP64 mode, 7 for half a Box-Muller pair and its step in the FP32 mode."""
    kind = case["kind"]
    if kind in ("book", "book_greeks"):
        # paths log-uniform in [2^a, 2^b], steps 252 x U(0.1, 5): the expected work of the drawn book
        a, b = case["log2_min"], case["log2_max"]
        paths = (2.0 ** b - 2.0 ** a) / ((b - a) * math.log(2.0))
        steps = case["options"] * paths * 252 * 2.55
        return {"bytes": 200.0 * case["options"], "flops": steps * (10.0 if kind == "book" else 22.0)}
    ps = float(case["paths"]) * case["steps"]
    anti = case.get("vr") == "antithetic" or kind == "asian"
    if kind in ("european", "greeks"):
        return {"bytes": 100.0, "flops": ps * (13.0 if anti else 25.0)}
    if kind in ("asian", "barrier"):
        return {"bytes": 100.0, "flops": ps * (18.0 if anti else 28.0)}
    if kind == "heston":
        return {"bytes": 100.0, "flops": ps * (36.0 if anti else 58.0)}
    if kind == "american":
        return {"bytes": ps * 32.0, "flops": ps * 45.0}
    if kind == "american_batch":
        n = ps * case["contracts"]
        return {"bytes": n * 16.0, "flops": n * 40.0}
    if kind == "strip":
        per = {"gbm": 5.0, "heston": 22.0, "qe": 60.0}[case["model"]]
        return {"bytes": 100.0, "flops": ps * per}
    if kind == "quick":
        return {"bytes": 100.0, "flops": ps * 5.0}
    # the adjoint: the forward step, its recompute and the Jacobian; states kept every 32 steps
    return {"bytes": ps * 16.0 / 32.0, "flops": ps * 150.0}


# ---- the same draws in 64 bits ---------------------------------------------

_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_M32 = 0xFFFFFFFF
_F64 = torch.float64


def _i64(x):
    x &= (1 << 64) - 1
    return x - (1 << 64) if x >> 63 else x


def _shr(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


def _rotl(x, k):
    return (x << k) | _shr(x, 64 - k)


class _Xoshiro:
    """xoshiro256++ streams, one per element of `s` (four int64 tensors)."""

    def __init__(self, s):
        self.s = list(s)

    @staticmethod
    def seeded(seeds):
        out, sm = [], seeds
        for _ in range(4):  # SplitMix64
            sm = sm + _i64(0x9E3779B97F4A7C15)
            z = (sm ^ _shr(sm, 30)) * _i64(0xBF58476D1CE4E5B9)
            z = (z ^ _shr(z, 27)) * _i64(0x94D049BB133111EB)
            out.append(z ^ _shr(z, 31))
        return _Xoshiro(out)

    def normal(self):
        s0, s1, s2, s3 = self.s
        r = _rotl(s0 + s3, 23) + s0
        t = s1 << 17
        s2 = s2 ^ s0
        s3 = s3 ^ s1
        s1 = s1 ^ s2
        s0 = s0 ^ s3
        self.s = [s0, s1, s2 ^ t, _rotl(s3, 45)]
        return _acklam(_shr(r, 11).to(_F64) * 2.0 ** -53)


def _poly(x, *c):
    y = torch.full_like(x, c[0])
    for a in c[1:]:
        y = y * x + a
    return y


def _acklam(p):
    """Acklam's rational approximation of the inverse normal, which defines the reference's normals."""
    eps = 2.0 ** -52
    p = p.clamp(eps, 1.0 - eps)
    q = p - 0.5
    r = q * q
    mid = q * _poly(r, -39.69683028665376, 220.9460984245205, -275.9285104469687, 138.357751867269, -30.66479806614716,
                    2.506628277459239) / _poly(r, -54.47609879822406, 161.5858368580409, -155.6989798598866,
                                               66.80131188771972, -13.28068155288572, 1.0)
    w = torch.sqrt(-2.0 * torch.log(torch.minimum(p, 1.0 - p)))
    tail = _poly(w, -7.784894002430293e-3, -0.3223964580411365, -2.400758277161838, -2.549732539343734,
                 4.374664141464968, 2.938163982698783) / _poly(w, 7.784695709041462e-3, 0.3224671290700398,
                                                               2.445134137142996, 3.754408661907416, 1.0)
    return torch.where(p < 0.02425, tail, torch.where(p <= 1.0 - 0.02425, mid, -tail))


def _philox(c0, c1, c2, c3, seed):
    k0, k1 = seed & _M32, (seed >> 32) & _M32
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = ((p1 >> 32) & _M32) ^ c1 ^ k0, p1 & _M32, ((p0 >> 32) & _M32) ^ c3 ^ k1, p0 & _M32
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return c0, c1, c2, c3


def _unif(r):
    return ((r >> 9).to(_F64) + 0.5) * 2.0 ** -23


def _pair(a, b):
    rad = torch.sqrt(-2.0 * torch.log(_unif(a)))
    ang = math.pi * ((b >> 9).to(_F64) * 2.0 ** -22 - 1.0)
    return rad * torch.cos(ang), rad * torch.sin(ang)


def _positive(call, s, k):
    return (s - k if call else k - s).clamp(min=0.0)


def _stats(x, df):
    n = x.numel()
    return np.array([df * float(x.mean())]), np.array([df * float(x.var()) ** 0.5 / n ** 0.5 if n > 1 else 0.0])


def _price32(x, df):
    p, s = _stats(x, df)
    return p[0], s[0]


def _exact_reference(case, t):
    """The FP64 engine's single options: a stream per sample, seeded seed + 7919 i."""
    kind, steps = case["kind"], case["steps"]
    anti = case.get("vr") == "antithetic" or kind == "asian"
    n = (case["paths"] + 1) // 2 if anti else case["paths"]
    rng = _Xoshiro.seeded(torch.arange(n, device=_DEV, dtype=torch.int64) * 7919 + t["seed"])
    S0, K, T, r, vol, call = t["spot"], t["strike"], t["expiry"], t["rate"], t["vol"], t["call"]
    dt, df = T / steps, math.exp(-r * T)
    signs = (1.0, -1.0) if anti else (1.0,)
    zero = torch.zeros(n, dtype=_F64, device=_DEV)
    if kind == "heston":
        legs = [[zero, zero + t["v0"]] for _ in signs]
        rc = math.sqrt(1.0 - t["rho"] ** 2)
        for _ in range(steps):
            z1, z2 = rng.normal(), rng.normal()
            zs = t["rho"] * z1 + rc * z2
            for leg, sg in zip(legs, signs):
                y, v = leg
                sq = torch.sqrt(v * dt)
                leg[0] = y + (r - 0.5 * v) * dt + sq * zs * sg
                leg[1] = (v + t["kappa"] * (t["theta"] - v) * dt + t["xi"] * sq * z1 * sg).clamp(min=0.0)
        x = sum(_positive(call, S0 * torch.exp(y), K) for y, _ in legs) / len(legs)
        p, s = _stats(x, df)
        return {"price": p, "stderr": s}
    a = r - 0.5 * vol * vol
    drift, diff = a * dt, vol * math.sqrt(dt)
    w = np.zeros(steps + 1)
    if kind == "asian":
        for u in _fixing_times(case, t):
            w[min(steps, int(math.floor(u / T * steps + 0.5)))] += 1.0
    up = case.get("style", "").startswith("up")
    sums = zero
    arith, geo, hit = [zero for _ in signs], [zero for _ in signs], [zero > 1.0 for _ in signs]
    for j in range(1, steps + 1):
        sums = sums + rng.normal()
        for k, sg in enumerate(signs):
            if kind == "barrier" or w[j]:
                y = drift * j + diff * sg * sums
                if kind == "barrier":
                    b = math.log(t["level"] / S0)
                    hit[k] = hit[k] | (y >= b if up else y <= b)
                else:
                    arith[k] = arith[k] + w[j] * torch.exp(y)
                    geo[k] = geo[k] + w[j] * y
    if kind == "asian":
        n_obs = w.sum()
        x = sum(_positive(call, S0 * s / n_obs, K) for s in arith) / 2.0
        if case["cv"]:
            y = sum(_positive(call, S0 * torch.exp(g / n_obs), K) for g in geo) / 2.0
            times = np.array(_fixing_times(case, t))
            m = math.log(S0) + a * times.mean()
            var = vol * vol * float(np.minimum.outer(times, times).sum()) / n_obs ** 2
            d2 = (m - math.log(K)) / math.sqrt(var)
            phi = lambda u: 0.5 * math.erfc(-u / math.sqrt(2.0))  # noqa: E731
            eg, sg = math.exp(m + 0.5 * var), 1.0 if call else -1.0
            e = sg * (eg * phi(sg * (d2 + math.sqrt(var))) - K * phi(sg * d2))
            xc, yc = x - x.mean(), y - y.mean()
            beta = float((xc * yc).sum() / (yc * yc).sum())
            x = x + beta * (e - y)
        p, s = _stats(x, df)
        return {"price": p, "stderr": s}
    ends = [S0 * torch.exp(a * T + diff * sg * sums) for sg in signs]
    if kind == "barrier":
        out = case["style"].endswith("out")
        x = sum(torch.where(~h if out else h, _positive(call, s, K), zero) for h, s in zip(hit, ends)) / len(ends)
        p, s = _stats(x, df)
        return {"price": p, "stderr": s}
    x = sum(_positive(call, s, K) for s in ends) / len(ends)
    p, se = _stats(x, df)
    if kind == "european":
        return {"price": p, "stderr": se}
    g = np.zeros(4)
    for sg, s in zip(signs, ends):
        one = torch.where(s > K, 1.0, 0.0) if call else torch.where(s < K, -1.0, 0.0)
        pv = df * _positive(call, s, K)
        z = sg * sums
        by_vol = one * s * (math.sqrt(dt) * z - vol * T)
        by_t = one * s * (a + vol * math.sqrt(dt) * z / (2.0 * T))
        for k, v in enumerate((df * one * s / S0, df * by_vol, r * pv - df * by_t, df * T * one * s - T * pv)):
            g[k] += float(v.mean()) / len(ends)
    return {"price": p, "stderr": se, "greeks": g}


def _stream_states(seed, count, draws):
    """The states of ONE xoshiro256++ stream after 0, draws, 2 draws, ... numbers: its update is linear over GF(2)."""
    def unpack(words):  # [n][4] -> [n][256] bits
        k = torch.arange(64, device=_DEV)
        return ((words[:, :, None] >> k) & 1).reshape(-1, 256).to(torch.float32)

    unit = torch.zeros(256, 4, dtype=torch.int64, device=_DEV)
    for j in range(256):
        unit[j, j // 64] = _i64(1 << (j % 64))
    g = _Xoshiro(unit.unbind(1))
    g.normal()
    step = unpack(torch.stack(g.s, 1))  # row j: the image of bit j
    jump, base, e = torch.eye(256, device=_DEV), step, draws
    while e:
        if e & 1:
            jump = torch.remainder(jump @ base, 2.0)
        base = torch.remainder(base @ base, 2.0)
        e >>= 1
    first = _Xoshiro.seeded(torch.tensor([_i64(seed)], device=_DEV))
    bits = unpack(torch.stack(first.s, 1))
    while bits.shape[0] < count:
        bits = torch.cat([bits, torch.remainder(bits @ jump, 2.0)])
        jump = torch.remainder(jump @ jump, 2.0)
    k = torch.arange(64, device=_DEV)
    words = (bits[:count].reshape(-1, 4, 64).to(torch.int64) << k).sum(2)
    return _Xoshiro(words.unbind(1))


def _least_squares(paths, put_strike, disc, degree):
    """Longstaff-Schwartz on paths[step-1][path]: each path's cash flow discounted to today and its payment step."""
    K, steps = put_strike, len(paths)
    v = (K - paths[-1]).clamp(min=0.0)
    tau = torch.full_like(v, float(steps))
    for t in range(steps - 1, 0, -1):
        v = v * disc
        s = paths[t - 1]
        itm = s < K
        x = (s / K - 1.0)[itm]
        if x.numel() < 3:
            continue
        A = torch.stack([x ** k for k in range(degree + 1)], 1)
        scale = A.abs().amax(0)
        A = A / scale
        beta = torch.linalg.solve(A.T @ A, A.T @ v[itm])
        now = torch.zeros_like(itm)
        now[itm] = (K - s[itm]) > A @ beta
        v = torch.where(now, K - s, v)
        tau = torch.where(now, float(t), tau)
    return v * disc, tau


def _exact_american(case, t):
    n, steps = case["paths"], case["steps"]
    rng = _stream_states(t["seed"], n, steps)
    dt = t["expiry"] / steps
    y, paths = torch.zeros(n, dtype=_F64, device=_DEV), []
    for _ in range(steps):
        y = y + (t["rate"] - 0.5 * t["vol"] ** 2) * dt + t["vol"] * math.sqrt(dt) * rng.normal()
        paths.append(t["spot"] * torch.exp(y))
    v, _ = _least_squares(paths, t["strike"], math.exp(-t["rate"] * dt), 2)
    p, s = _stats(v, 1.0)
    return {"price": p, "stderr": s}


def _exact_american_batch(case, seed):
    spots, vols, stream = _puts(case, seed)
    steps, dt = case["steps"], 1.0 / 50.0
    disc = math.exp(-0.06 * dt)
    idx = torch.arange(case["paths"], device=_DEV, dtype=torch.int64)
    out = {"price": [], "stderr": [], "delta": []}
    for c, (s0, vol) in enumerate(zip(spots, vols)):
        y, paths = torch.zeros(case["paths"], dtype=_F64, device=_DEV), []
        for b in range(0, steps, 4):
            r = _philox(b // 4, idx, c, 0x4C534D31, stream)
            for z in (_pair(r[0], r[1]) + _pair(r[2], r[3]))[:steps - b]:
                y = y + (0.06 - 0.5 * vol * vol) * dt + vol * math.sqrt(dt) * z
                paths.append(s0 * torch.exp(y))
        v, tau = _least_squares(paths, 40.0, disc, 3)
        p, s = _price32(v, 1.0)
        # a cash flow v = (K - S) disc^tau moves with the spot by -S disc^tau / S0
        d = torch.where(v > 0.0, -(40.0 * disc ** tau - v) / s0, 0.0)
        for key, val in (("price", p), ("stderr", s), ("delta", float(d.mean()))):
            out[key].append(val)
    return {k: np.array(v) for k, v in out.items()}


def _exact_strip(case, t):
    steps, model = case["steps"], case.get("model", "gbm")
    anti = case.get("vr") == "antithetic"
    n = (case["paths"] + 1) // 2 if anti else case["paths"]
    idx = torch.arange(n, device=_DEV, dtype=torch.int64)
    dt, r = t["expiry"] / steps, t["rate"]
    df, sq = math.exp(-r * t["expiry"]), math.sqrt(dt)
    signs = (1.0, -1.0) if anti else (1.0,)
    zero = torch.zeros(n, dtype=_F64, device=_DEV)
    if model == "gbm":
        w = zero
        for b in range(0, steps, 4):
            q = _philox(b // 4, idx, 0, 0x53545250, t["seed"])
            for z in (_pair(q[0], q[1]) + _pair(q[2], q[3]))[:steps - b]:
                w = w + z
        ys = [(r - 0.5 * t["vol"] ** 2) * t["expiry"] + sg * t["vol"] * sq * w for sg in signs]
    else:
        legs = [[zero, zero + t["v0"]] for _ in signs]
        qe = _QeStep(t, dt, 0.0)
        for b in range(0, steps, 2):
            q = _philox(b // 2, idx, 0, 0x53545250, t["seed"])
            for k in range(min(2, steps - b)):
                if model == "heston":
                    z1, z2 = _pair(q[2 * k], q[2 * k + 1])
                    zs = t["rho"] * z1 + math.sqrt(1.0 - t["rho"] ** 2) * z2
                else:
                    u = _unif(q[2 * k])
                    zv, zx = torch.special.ndtri(u), torch.special.ndtri(_unif(q[2 * k + 1]))
                for leg, sg in zip(legs, signs):
                    y, v = leg
                    if model == "heston":
                        sv = torch.sqrt(v) * sq
                        leg[0] = y + (r - 0.5 * v) * dt + sv * zs * sg
                        leg[1] = (v + t["kappa"] * (t["theta"] - v) * dt + t["xi"] * sv * z1 * sg).clamp(min=0.0)
                    else:
                        d0 = torch.zeros(0, 1, dtype=_F64, device=_DEV)
                        yn, vn = qe(_Dual(y, d0), _Dual(v, d0), u if sg > 0 else 1.0 - u, zv * sg, zx * sg)
                        leg[0], leg[1] = yn.v, vn.v
        ys = [y for y, _ in legs]
    ends = [t["spot"] * torch.exp(y) for y in ys]
    strikes = _strikes(case, t) if case["kind"] == "strip" else [t["strike"]]
    got = [_price32(sum(_positive(t["call"], s, k) for s in ends) / len(ends), df) for k in strikes]
    return {"price": np.array([p for p, _ in got]), "stderr": np.array([s for _, s in got])}


class _Dual:
    """A value per sample and its derivatives along k parameters (k = 0: the value alone)."""

    def __init__(self, v, d):
        self.v, self.d = v, d

    def __add__(self, o):
        return _Dual(self.v + o.v, self.d + o.d) if isinstance(o, _Dual) else _Dual(self.v + o, self.d)

    def __mul__(self, o):
        return _Dual(self.v * o.v, self.d * o.v + o.d * self.v) if isinstance(o, _Dual) else _Dual(self.v * o, self.d * o)

    def __neg__(self):
        return _Dual(-self.v, -self.d)

    def __sub__(self, o):
        return self + (-o)

    def __rsub__(self, o):
        return -self + o

    def __truediv__(self, o):
        return self * (o.inv() if isinstance(o, _Dual) else 1.0 / o)

    def __rtruediv__(self, o):
        return self.inv() * o

    __radd__, __rmul__ = __add__, __mul__

    def inv(self):
        i = 1.0 / self.v
        return _Dual(i, -self.d * (i * i))

    def exp(self):
        e = torch.exp(self.v)
        return _Dual(e, self.d * e)

    def log(self):
        return _Dual(torch.log(self.v), self.d / self.v)

    def sqrt(self):
        r = torch.sqrt(self.v)
        return _Dual(r, self.d * torch.where(r > 0.0, 0.5 / r, 0.0))

    def where(self, mask, o):
        return _Dual(torch.where(mask, self.v, o.v), torch.where(mask, self.d, o.d))

    def at(self, i):  # the parameter of each sample
        return _Dual(self.v[i], self.d[:, i])


def _phi(x):
    return torch.exp(-0.5 * x * x) / math.sqrt(2.0 * math.pi)


class _QeStep:
    """Andersen's quadratic-exponential step, the branches blended by a smoothstep over psi = 1.5 -+ band."""

    def __init__(self, p, dt, band):
        self.p, self.band = p, band
        k, th, x, rho = p["kappa"], p["theta"], p["xi"], p["rho"]
        one = k * 0.0 + 1.0
        self.e = (k * -dt).exp() if isinstance(k, _Dual) else math.exp(-k * dt)
        self.c1 = x * x * self.e * (one - self.e) / k
        self.c2 = th * x * x * (one - self.e) * (one - self.e) / (k * 2.0)
        kr = (k * rho / x - 0.5) * (0.5 * dt)
        self.c0 = p["rate"] * dt - rho * k * th * dt / x
        self.k1, self.k2 = kr - rho / x, kr + rho / x
        self.k34 = (one - rho * rho) * (0.5 * dt)

    def __call__(self, y, v, u, zv, zx):
        m = (v - self.p["theta"]) * self.e + self.p["theta"]
        psi = (v * self.c1 + self.c2) / (m * m)
        quad, expo = psi.v <= 1.5 + self.band, psi.v > 1.5 - self.band
        t = 2.0 / psi
        b2 = (t - 1.0) + _Dual(t.v.clamp(min=1.0), t.d * (t.v > 1.0)).sqrt() * \
            _Dual((t.v - 1.0).clamp(min=0.0), t.d * (t.v > 1.0)).sqrt()
        bz = _Dual(b2.v.clamp(min=1e-30), b2.d).sqrt() + zv
        vq = m / (b2 + 1.0) * bz * bz
        q = 1.0 - (psi - 1.0) / (psi + 1.0)
        dead = u <= 1.0 - q.v
        lg = q.log() - torch.log1p(-u)
        ve = m * lg / q
        ve = _Dual(torch.where(dead, 0.0, ve.v), torch.where(dead, 0.0, ve.d))
        vn = vq.where(~expo, ve)
        if self.band:
            s = (psi - (1.5 - self.band)) / (2.0 * self.band)
            w = s * s * (3.0 - s * 2.0)
            vn = (vq + w * (ve - vq)).where(quad & expo, vn)
        yn = y + self.c0 + v * self.k1 + vn * self.k2 + ((v + vn) * self.k34).sqrt() * zx
        return yn, vn


def _exact_adjoint(case, t):
    n, steps, T = case["paths"], case["steps"], t["expiry"]
    eye = torch.eye(7, dtype=_F64, device=_DEV)[:, :, None]
    names = ("spot", "rate", "v0", "kappa", "theta", "xi", "rho")
    p = {k: _Dual(torch.tensor(t[k], dtype=_F64, device=_DEV), eye[i]) for i, k in enumerate(names)}
    sign = 1.0 if t["call"] else -1.0
    sums, means = [], []
    for lo in range(0, n, 1 << 18):
        idx = torch.arange(lo, min(n, lo + (1 << 18)), device=_DEV, dtype=torch.int64)
        zero = torch.zeros(idx.numel(), dtype=_F64, device=_DEV)
        y, v = _Dual(zero, torch.zeros(7, 1, dtype=_F64, device=_DEV)), p["v0"] + zero
        avg = y
        qe = _QeStep(p, T / steps, 0.05)
        for b in range(0, steps, 2):
            q = _philox(b // 2, idx, 0, 0x41444A31, t["seed"])
            for k in range(min(2, steps - b)):
                u = _unif(q[2 * k])
                y, v = qe(y, v, u, torch.special.ndtri(u), torch.special.ndtri(_unif(q[2 * k + 1])))
                if case["asian"]:
                    avg = avg + y.exp()
        und = p["spot"] * (avg * (1.0 / steps) if case["asian"] else y.exp())
        x = (und - t["strike"]) * sign
        x = _Dual(x.v.clamp(min=0.0), x.d * (x.v > 0.0)) * (p["rate"] * -T).exp()
        rows = torch.cat([x.v[None], x.d])
        sums.append(torch.stack([rows.sum(1), (rows * rows).sum(1)]))
    s = torch.stack(sums).sum(0)
    mean = s[0] / n
    se = torch.sqrt((s[1] - s[0] * s[0] / n).clamp(min=0.0) / (n - 1.0) / n)
    mean, se = mean.cpu().numpy(), se.cpu().numpy()
    return {"price": mean[:1], "stderr": se[:1], "greeks": mean[1:], "greeks_se": se[1:]}


def _exact_book(case, seed):
    """The book's options in flat vectors, a few million samples at a time; with Greeks, barriers by one-step survival
    (Glasserman and Staum, 2001) as the engine prices them then."""
    entries, stream = _book(case, seed)
    greeks, anti = case["kind"] == "book_greeks", case["vr"] == "antithetic"
    k, n = 4 if greeks else 0, len(entries)
    samples = [(e["paths"] + 1) // 2 if anti else e["paths"] for e in entries]
    if sum(m * e["steps"] for m, e in zip(samples, entries)) > (4e9 if greeks else 2.5e10):
        return None
    col = {f: torch.tensor([e[f] for e in entries], dtype=_F64, device=_DEV)
           for f in ("s0", "strike", "vol", "rate", "expiry", "steps", "level")}
    one = torch.eye(k, dtype=_F64, device=_DEV)[:, :, None].expand(k, k, n) if k else \
        torch.zeros(4, 0, n, dtype=_F64, device=_DEV)
    par = {f: _Dual(col[f], one[i]) for i, f in enumerate(("s0", "vol", "rate", "expiry"))}
    out = torch.zeros(1 + k, n, dtype=_F64, device=_DEV)
    out2 = torch.zeros_like(out)
    cap = (1 << 19) if greeks else (1 << 22)
    for kind in ("european", "asian", "barrier"):
        todo = sorted((i for i in range(n) if entries[i]["kind"] == kind), key=lambda i: -entries[i]["steps"])
        pieces = [(i, lo, min(samples[i], lo + cap)) for i in todo for lo in range(0, samples[i], cap)]
        while pieces:
            part, size = [], 0
            while pieces and (not part or size + pieces[0][2] - pieces[0][1] <= cap):
                part.append(pieces.pop(0))
                size += part[-1][2] - part[-1][1]
            opt = torch.cat([torch.full((hi - lo,), i, device=_DEV, dtype=torch.int64) for i, lo, hi in part])
            idx = torch.cat([torch.arange(lo, hi, device=_DEV, dtype=torch.int64) for _, lo, hi in part])
            x = _book_samples(kind, entries[part[0][0]]["steps"], opt, idx, col, par, stream, greeks, anti)
            for row in range(1 + k):
                out[row].index_add_(0, opt, x[row])
                out2[row].index_add_(0, opt, x[row] * x[row])
    m = torch.tensor(samples, dtype=_F64, device=_DEV)
    mean = out / m
    se = torch.sqrt((out2 - out * out / m).clamp(min=0.0) / (m - 1.0) / m)
    mean, se = mean.cpu().numpy(), se.cpu().numpy()
    res = {"price": mean[0], "stderr": se[0]}
    if greeks:
        for row, g, sg in ((1, "delta", 1.0), (2, "vega", 1.0), (3, "rho", 1.0), (4, "theta", -1.0)):
            res[g], res[g + "_se"] = sg * mean[row], se[row]
    return res


def _book_samples(kind, max_steps, opt, idx, col, par, stream, greeks, anti):
    """Discounted payoff of each sample and its derivatives, as rows."""
    s0, vol, rate, T = (par[f].at(opt) for f in ("s0", "vol", "rate", "expiry"))
    steps, strike = col["steps"][opt], col["strike"][opt]
    dt = T * (1.0 / steps)
    alpha, beta = (rate - vol * vol * 0.5) * dt, vol * dt.sqrt()
    zero = _Dual(torch.zeros_like(strike), torch.zeros(s0.d.shape[0], 1, dtype=_F64, device=_DEV))
    survival = kind == "barrier" and greeks
    bar = -(s0 * (1.0 / col["level"][opt])).log()
    signs = (1.0, -1.0) if anti else (1.0,)
    y, acc = [zero for _ in signs], [zero + 1.0 if survival else zero for _ in signs]
    dead, w = [torch.zeros_like(opt, dtype=torch.bool) for _ in signs], torch.zeros_like(strike)
    for q in range(0, max_steps, 4):
        r = _philox(q // 4, idx, 0, opt, stream)
        zs = [_unif(a) for a in r] if survival else _pair(r[0], r[1]) + _pair(r[2], r[3])
        for j, z in enumerate(zs[:max_steps - q]):
            on = steps > q + j
            if kind == "european":
                w = w + torch.where(on, z, 0.0)
                continue
            for leg, sg in enumerate(signs):
                if not survival:
                    yn = y[leg] + alpha + beta * (z * sg)
                    y[leg] = yn.where(on, y[leg])
                    if kind == "asian":
                        acc[leg] = (acc[leg] + yn.exp()).where(on, acc[leg])
                    else:
                        dead[leg] = dead[leg] | (on & (yn.v >= bar.v))
                    continue
                u = z if sg > 0 else 1.0 - z
                h = (bar - y[leg] - alpha) / beta
                h = _Dual(h.v.clamp(min=-37.0), h.d)
                p = _Dual(torch.special.ndtr(h.v), h.d * _phi(h.v))
                v = p * u
                zeta = torch.where(v.v <= 0.5, torch.special.ndtri(v.v.clamp(min=1e-300)),
                                   -torch.special.ndtri((1.0 - v.v).clamp(min=1e-300)))
                zeta = _Dual(zeta, v.d / _phi(zeta))
                yn = y[leg] + alpha + beta * zeta
                y[leg], acc[leg] = yn.where(on, y[leg]), (acc[leg] * p).where(on, acc[leg])
    rows = 0.0
    for leg, sg in enumerate(signs):
        if kind == "european":
            y[leg] = alpha * steps + beta * (w * sg)
        s = s0 * (acc[leg] * (1.0 / steps) if kind == "asian" else y[leg].exp())
        x = s - strike
        x = _Dual(torch.where(dead[leg], 0.0, x.v.clamp(min=0.0)), x.d * ((x.v > 0.0) & ~dead[leg]))
        if survival:
            x = x * acc[leg]
        x = x * (-(rate * T)).exp()
        rows = rows + torch.cat([x.v[None], x.d.expand(x.d.shape[0], x.v.numel())]) / len(signs)
    return rows


def exact(case, seed):
    kind = case["kind"]
    if kind in ("book", "book_greeks"):
        return _exact_book(case, seed)
    if kind == "american_batch":
        if case["contracts"] * case["paths"] * case["steps"] > 4e9:
            return None
        return _exact_american_batch(case, seed)
    t = _terms(case, seed)
    if kind in ("strip", "quick"):
        return _exact_strip(case, t)
    if kind == "american":
        return _exact_american(case, t)
    if kind == "adjoint":
        return _exact_adjoint(case, t)
    return _exact_reference(case, t)
