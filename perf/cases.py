"""Performance cases of the engine: what its users ask of it, through the
public Python entry points, from one small European price to a 256-contract
book. Monte-Carlo inputs are a contract, a model and a seed, so a state is a
few Python objects; each seed moves the market a little and gives the call
its own random stream.

`exact` restates every case in 64-bit torch arithmetic on the same
Philox4x32-10 + Box-Muller normals.
"""
import math
import random

import numpy as np
import torch

import kontracts_gb300 as kx
from kontracts_gb300 import calibration

ASSET = "S"
HESTON = (0.04, 2.0, 0.04, 0.3, -0.5)  # v0, kappa, theta, sigma_v, rho


def listed():
    return [
        # a single quote with the API's default arguments: the call's fixed cost
        {"name": "european_default", "kind": "price", "product": "european", "model": "gbm", "precision": "fp32",
         "n": 100_000, "spy": 50, "maturity": 1.0, "s0": 100.0, "strike": 100.0, "sigma": 0.2, "rate": 0.05},
        # the same contract in the reference's own precision, one million paths
        {"name": "european_fp64", "kind": "price", "product": "european", "model": "gbm", "precision": "fp64",
         "n": 1_000_000, "spy": 1, "maturity": 1.0, "s0": 100.0, "strike": 100.0, "sigma": 0.2, "rate": 0.05},
        # the benchmark's daily-monitored knock-out at full size
        {"name": "up_and_out_4m", "kind": "price", "product": "up_and_out", "model": "gbm", "precision": "fp32",
         "n": 4_000_000, "spy": 365, "maturity": 1.0, "s0": 180.0, "strike": 100.0, "barrier": 200.0, "sigma": 0.25,
         "rate": 0.05},
        # an arithmetic Asian with a maturity between grid points and an odd path count
        {"name": "asian", "kind": "price", "product": "asian", "model": "gbm", "precision": "fp32", "n": 500_003,
         "spy": 252, "maturity": 1.3, "s0": 100.0, "strike": 105.0, "sigma": 0.3, "rate": 0.03},
        # a contract whose acquisition depends on the price (down-and-in put)
        {"name": "knock_in", "kind": "price", "product": "knock_in", "model": "gbm", "precision": "fp32",
         "n": 1_000_001, "spy": 252, "maturity": 0.75, "s0": 100.0, "strike": 100.0, "barrier": 90.0, "sigma": 0.25,
         "rate": 0.02},
        # a strike ladder at three maturities on one Heston simulation
        {"name": "heston_book", "kind": "heston_book", "n": 2_000_000, "spy": 252, "strikes": 32, "maturities": 3},
        # bump-and-reprice Greeks of a path-dependent contract (seven reprices)
        {"name": "greeks_asian", "kind": "greeks", "product": "asian", "model": "gbm", "precision": "fp32",
         "n": 200_000, "spy": 252, "maturity": 1.0, "s0": 100.0, "strike": 100.0, "sigma": 0.2, "rate": 0.05},
        # price and all seven Heston sensitivities by the pathwise adjoint
        {"name": "adjoint_heston", "kind": "adjoint", "product": "european", "model": "heston", "n": 2_000_000,
         "spy": 252, "maturity": 1.0, "s0": 100.0, "strike": 100.0, "sigma": 0.2, "rate": 0.05},
        # an American put by Longstaff-Schwartz
        {"name": "american_put", "kind": "american", "precision": "fp32", "basis": "laguerre", "n_basis": 4,
         "n": 1_000_000, "dates": 50, "maturity": 1.0, "s0": 36.0, "strike": 40.0, "sigma": 0.2, "rate": 0.06},
        # an uneven book revalued through its captured graph
        {"name": "book_256", "kind": "book", "contracts": 256, "n_lo": 65_536, "n_hi": 1_048_576, "spy": 252},
        # a knock-out call on a basket of five correlated assets
        {"name": "basket_5", "kind": "basket", "factors": 5, "n": 1_000_000, "spy": 252, "maturity": 1.0,
         "strike": 100.0, "barrier": 130.0},
        # one generation of a Heston calibration in its default precision
        {"name": "calibration_generation", "kind": "calibration", "candidates": 40, "quotes": 3, "n": 3_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("price", "price", "price", "heston_book", "greeks", "adjoint", "american", "book", "basket",
                       "calibration"))
    market = {"maturity": round(rng.uniform(0.25, 2.0), 3), "s0": 100.0, "strike": round(rng.uniform(80, 120), 2),
              "sigma": round(rng.uniform(0.1, 0.5), 3), "rate": round(rng.uniform(0.0, 0.06), 4)}
    if kind == "price":
        c = {"kind": kind, "product": rng.choice(("european", "up_and_out", "asian", "knock_in")), "model": "gbm",
             "precision": "fp32", "n": _log_int(rng, 10_000, 4_000_000), "spy": rng.choice((50, 252, 365)), **market}
        if rng.random() < 0.25:
            c["precision"] = "fp64"
            c["n"] = _log_int(rng, 10_000, 1_000_000 if c["product"] == "european" else 100_000)
        elif rng.random() < 0.25:
            c["model"], c["product"], c["n"] = "heston", "european", _log_int(rng, 10_000, 1_000_000)
        if c["product"] == "up_and_out":
            c["barrier"] = round(100.0 * rng.uniform(1.1, 1.5), 2)
            c["strike"] = round(rng.uniform(80, 105), 2)
        elif c["product"] == "knock_in":
            c["barrier"] = round(100.0 * rng.uniform(0.75, 0.95), 2)
            c["strike"] = round(rng.uniform(95, 120), 2)
        return c
    if kind == "heston_book":
        return {"kind": kind, "n": _log_int(rng, 50_000, 2_000_000), "spy": 252, "strikes": rng.randint(3, 32),
                "maturities": rng.randint(1, 3)}
    if kind == "greeks":
        return {"kind": kind, "product": rng.choice(("european", "asian")), "model": "gbm", "precision": "fp32",
                "n": _log_int(rng, 20_000, 500_000), "spy": rng.choice((50, 252)), **market}
    if kind == "adjoint":
        c = {"kind": kind, "product": "european", "model": "heston", "n": _log_int(rng, 50_000, 2_000_000), "spy": 252,
             **market, "maturity": round(rng.uniform(0.25, 1.0), 3)}
        if rng.random() < 0.6:
            c["model"], c["product"] = "gbm", rng.choice(("asian", "up_and_out"))
            c["barrier"] = round(100.0 * rng.uniform(1.2, 1.5), 2)
            c["strike"] = round(rng.uniform(80, 105), 2)
        return c
    if kind == "american":
        fp64 = rng.random() < 0.25
        return {"kind": kind, "precision": "fp64" if fp64 else "fp32", "basis": rng.choice(("monomial", "laguerre")),
                "n_basis": rng.choice((3, 4)), "n": _log_int(rng, 20_000, 200_000 if fp64 else 1_000_000),
                "dates": rng.choice((12, 25, 50, 100)), "maturity": round(rng.uniform(0.5, 2.0), 3),
                "s0": round(rng.uniform(36, 44), 2), "strike": 40.0, "sigma": round(rng.uniform(0.2, 0.4), 3),
                "rate": 0.06}
    if kind == "book":
        return {"kind": kind, "contracts": _log_int(rng, 8, 200), "n_lo": 16_384, "n_hi": 524_288,
                "spy": rng.choice((50, 252))}
    if kind == "basket":
        return {"kind": kind, "factors": rng.randint(2, 5), "n": _log_int(rng, 20_000, 1_000_000), "spy": 252,
                "maturity": round(rng.uniform(0.25, 1.0), 3), "strike": round(rng.uniform(90, 110), 2),
                "barrier": round(rng.uniform(120, 150), 2)}
    return {"kind": "calibration", "candidates": rng.choice((6, 16, 24, 40)), "quotes": rng.randint(1, 3),
            "n": _log_int(rng, 1_000, 3_000)}


# --- the inputs of a case, from its seed ---------------------------------------------------------


def _market(case, seed):
    """The case's market moved by up to a per cent, and the stream of its paths."""
    rng = random.Random(seed)
    return {"s0": case["s0"] * rng.uniform(0.99, 1.01), "sigma": case["sigma"] * rng.uniform(0.98, 1.02),
            "seed": rng.getrandbits(40)}


def _heston_market(seed, s0=100.0):
    rng = random.Random(seed)
    return {"s0": s0 * rng.uniform(0.99, 1.01), "v0": HESTON[0] * rng.uniform(0.95, 1.05), "kappa": HESTON[1],
            "theta": HESTON[2], "sigma_v": HESTON[3], "rho": HESTON[4], "seed": rng.getrandbits(40)}


def _heston_model(p, rate):
    return kx.heston(p["s0"], p["v0"], p["kappa"], p["theta"], p["sigma_v"], p["rho"], rate, asset=ASSET,
                     scheme="full_truncation")


def _asian_call(strike, maturity):
    return kx.scale((kx.average(kx.S(ASSET)) - strike).clip(0.0), kx.one()) @ kx.at(maturity)


def _contract(case):
    k, t = case["strike"], case["maturity"]
    if case["product"] == "european":
        return kx.european_call(ASSET, k, t)
    if case["product"] == "up_and_out":
        return kx.up_and_out_call(ASSET, k, case["barrier"], t)
    if case["product"] == "asian":
        return _asian_call(k, t)
    return kx.when(kx.S(ASSET) <= case["barrier"], kx.european_put(ASSET, k, t))  # knock_in


def _heston_ladder(case):
    """(strike, maturity) of the ladder: evenly spaced strikes in [80, 120], maturities 0.5, 1, 2."""
    m = max(1, case["strikes"] - 1)
    return [(80.0 + 40.0 * i / m, t) for t in (0.5, 1.0, 2.0)[:case["maturities"]] for i in range(case["strikes"])]


def _book(case, seed):
    """A 50 / 30 / 20 mix of European, up-and-out and Asian calls with uneven paths and maturities."""
    rng = random.Random(seed)
    n = case["contracts"]
    kinds = ["up_and_out"] * round(0.3 * n) + ["asian"] * round(0.2 * n)
    kinds += ["european"] * (n - len(kinds))
    rng.shuffle(kinds)
    return [{"product": p, "s0": 100.0, "strike": rng.uniform(80, 120), "sigma": rng.uniform(0.1, 0.5), "rate": 0.03,
             "barrier": 100.0 * rng.uniform(1.1, 1.5), "maturity": rng.uniform(0.25, 2.0),
             "n": _log_int(rng, case["n_lo"], case["n_hi"]), "seed": rng.getrandbits(40)} for p in kinds]


def _basket(case, seed):
    rng = random.Random(seed)
    k = case["factors"]
    return {"s0": [100.0 * rng.uniform(0.99, 1.01) for _ in range(k)], "sigma": [0.15 + 0.05 * i for i in range(k)],
            "corr": [[1.0 if i == j else 0.4 for j in range(k)] for i in range(k)], "rate": 0.03,
            "seed": rng.getrandbits(40)}


def _calibration(case, seed):
    """Quotes near the prices of the usual parameters, and a population around them in the search box."""
    rng = random.Random(seed)
    lo, hi = calibration.HESTON_LOWER, calibration.HESTON_UPPER
    pop = [[min(max(x + 0.1 * (b - a) * rng.gauss(0, 1), a), b) for x, a, b in zip(HESTON, lo, hi)]
           for _ in range(case["candidates"])]
    quotes = [(s * rng.uniform(0.99, 1.01), p * rng.uniform(0.97, 1.03))
              for s, p in ((90.0, 5.0), (100.0, 10.4), (110.0, 17.5))[:case["quotes"]]]
    return {"quotes": quotes, "population": pop, "rate": 0.05, "strike": 100.0, "maturity": 1.0}


# --- one pass through the public entry points -----------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("price", "greeks", "adjoint"):
        contract = _contract(case)
        contract.plan()  # compiled once, as a program that prices a contract repeatedly keeps it
        if case["model"] == "heston":
            p = _heston_market(seed, case["s0"])
            model = _heston_model(p, case["rate"])
        else:
            p = _market(case, seed)
            model = kx.GBM(s0=p["s0"], sigma=p["sigma"], r=case["rate"], asset=ASSET)
        return {"case": case, "contract": contract, "model": model, "seed": p["seed"]}
    if kind == "heston_book":
        p = _heston_market(seed)
        book = [kx.european_call(ASSET, k, t) for k, t in _heston_ladder(case)]
        for c in book:
            c.plan()
        return {"case": case, "contracts": book, "model": _heston_model(p, 0.05), "seed": p["seed"]}
    if kind == "american":
        p = _market(case, seed)
        put = kx.scale((kx.const_(case["strike"]) - kx.S(ASSET)).clip(0.0), kx.one())
        put.plan()
        return {"case": case, "contract": put, "dates": _dates(case), "seed": p["seed"],
                "model": kx.GBM(s0=p["s0"], sigma=p["sigma"], r=case["rate"], asset=ASSET)}
    if kind == "book":
        items = _book(case, seed)
        return {"case": case, "book": kx.Book([_contract(b) for b in items],
                                              [kx.GBM(s0=b["s0"], sigma=b["sigma"], r=b["rate"], asset=ASSET)
                                               for b in items],
                                              [b["n"] for b in items], [b["seed"] for b in items],
                                              steps_per_year=case["spy"])}
    if kind == "basket":
        p = _basket(case, seed)
        names = ["A%d" % i for i in range(case["factors"])]
        level = kx.S(names[0])
        for a in names[1:]:
            level = level + kx.S(a)
        level = level / float(case["factors"])
        call = kx.scale((level - case["strike"]).clip(0.0), kx.one()) @ kx.at(case["maturity"])
        contract = kx.until(level >= case["barrier"], call)
        contract.plan()
        model = kx.CorrelatedGbmN([(a, s, p["rate"], v) for a, s, v in zip(names, p["s0"], p["sigma"])], p["corr"],
                                  rate=p["rate"])
        return {"case": case, "contract": contract, "model": model, "seed": p["seed"]}
    p = _calibration(case, seed)
    contract = kx.european_call("underlying", p["strike"], p["maturity"])
    contract.plan()
    return {"case": case, "contract": contract, **p}


def _dates(case):
    n = case["dates"]
    return [case["maturity"] * i / n for i in range(1, n + 1)]


def _result(r, precision):
    out = {"price": r.price, "sample_std": r.sample_std, "std_error": r.std_error}
    return {k: np.float64(v) for k, v in out.items()} if precision == "fp64" else out


GREEKS = ("price", "delta", "gamma", "vega", "rho", "price_se", "delta_se", "gamma_se", "vega_se", "rho_se")
SENS = {"gbm": ("s0", "sigma", "r"), "heston": ("s0", "v0", "kappa", "theta", "sigma_v", "rho", "r")}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "price":
        r = state["contract"].price(state["model"], n_paths=case["n"], seed=state["seed"], steps_per_year=case["spy"],
                                    precision=case["precision"])
        return _result(r, case["precision"])
    if kind == "heston_book":
        rs = kx.price_batch(state["contracts"], state["model"], n_paths=case["n"], seed=state["seed"],
                            steps_per_year=case["spy"])
        return _columns(rs)
    if kind == "greeks":
        g = state["contract"].greeks(state["model"], n_paths=case["n"], seed=state["seed"],
                                     steps_per_year=case["spy"], bumps=(1e-2, 1e-2, 1e-2), relative=True,
                                     precision=case["precision"])
        return {k: getattr(g, k) for k in GREEKS}
    if kind == "adjoint":
        s = state["contract"].adjoint(state["model"], n_paths=case["n"], seed=state["seed"],
                                      steps_per_year=case["spy"])
        out = {"price": s.price, "price_se": s.price_se}
        for q in SENS[case["model"]]:
            out["d_" + q], out["se_" + q] = getattr(s, "d_" + q), getattr(s, "se_" + q)
        return out
    if kind == "american":
        r = state["contract"].price_american(state["model"], state["dates"], n_paths=case["n"], seed=state["seed"],
                                             n_basis=case["n_basis"], basis=case["basis"],
                                             precision=case["precision"])
        return {"price": r.price, "sample_std": r.sample_std, "std_error": r.std_error}
    if kind == "book":
        return _columns(state["book"].price())
    if kind == "basket":
        r = state["contract"].price(state["model"], n_paths=case["n"], seed=state["seed"], steps_per_year=case["spy"])
        return _result(r, "fp32")
    return calibration.heston_objective(state["contract"], state["quotes"], state["population"], state["rate"],
                                        case["n"])


def _columns(results):
    """The results of FP32 paths, one array a column."""
    return {"price": np.array([r.price for r in results], dtype=np.float32),
            "sample_std": np.array([r.sample_std for r in results], dtype=np.float32),
            "std_error": np.array([r.std_error for r in results], dtype=np.float32)}


# --- what a pass cannot do without ----------------------------------------------------------------

NORMAL = 28  # operations of one normal: a quarter of Philox4x32-10 (20 of its 80), half a Box-Muller pair (8)
GBM_STEP, HESTON_STEP, TANGENT = 3, 15, 25


def _steps(case, maturity=None, forced=False):
    t = case["maturity"] if maturity is None else maturity
    fine = forced or case.get("product") in ("up_and_out", "asian", "knock_in")
    return math.ceil(t * case["spy"]) if fine else 1


def _alive(s0, barrier, sigma, rate, maturity):
    """Mean share of its steps that an up-and-out path takes (continuous monitoring, reflection principle)."""
    b, mu, total = math.log(barrier / s0), rate - 0.5 * sigma * sigma, 0.0
    if b <= 0:
        return 0.0
    cdf = lambda x: 0.5 * math.erfc(-x / math.sqrt(2.0))  # noqa: E731
    for i in range(64):
        t = maturity * (i + 0.5) / 64
        sd = sigma * math.sqrt(t)
        total += cdf((b - mu * t) / sd) - math.exp(2 * mu * b / sigma ** 2) * cdf((-b - mu * t) / sd)
    return total / 64


def _path_steps(case):
    steps = _steps(case, forced=case.get("model") == "heston")
    if case["product"] == "up_and_out":
        steps *= _alive(case["s0"], case["barrier"], case["sigma"], case["rate"], case["maturity"])
    return case["n"] * max(1.0, steps)


def work(case):
    kind = case["kind"]
    if kind in ("price", "greeks"):
        per = 2 * NORMAL + HESTON_STEP if case["model"] == "heston" else NORMAL + GBM_STEP
        if case["product"] == "asian":
            per += 3  # the spot of every step in the average
        flops = _path_steps(case) * per
        if kind == "greeks":  # the seven paths share their normals
            flops += 6 * _path_steps(case) * (per - NORMAL)
        return {"bytes": 80, "flops": flops}
    if kind == "heston_book":
        steps = math.ceil((0.5, 1.0, 2.0)[case["maturities"] - 1] * case["spy"])
        return {"bytes": 12 * case["strikes"] * case["maturities"],
                "flops": case["n"] * (steps * (2 * NORMAL + HESTON_STEP) + 3 * case["strikes"] * case["maturities"])}
    if kind == "adjoint":
        steps = case["n"] * _steps(case, forced=case["model"] == "heston")
        per = 2 * NORMAL + HESTON_STEP + 2 * TANGENT if case["model"] == "heston" else NORMAL + GBM_STEP + 12
        return {"bytes": 128, "flops": steps * per}
    if kind == "american":
        size = 8 if case["precision"] == "fp64" else 4
        cells = case["n"] * case["dates"]  # every spot is kept for the backward pass: written once, read once
        m = case["n_basis"]
        return {"bytes": 2 * size * cells, "flops": cells * (NORMAL + GBM_STEP + 2 * m + m * (m + 3))}
    if kind == "book":
        flops = 0.0
        for b in _book(case, 0):
            flops += _path_steps({**b, "spy": case["spy"]}) * (NORMAL + GBM_STEP + 3 * (b["product"] == "asian"))
        return {"bytes": 12 * case["contracts"], "flops": flops}
    if kind == "basket":
        k = case["factors"]
        return {"bytes": 24, "flops": case["n"] * math.ceil(case["maturity"] * case["spy"])
                * (k * (NORMAL + GBM_STEP) + k * (k + 1) + 2 * k)}
    prices = case["candidates"] * case["quotes"]  # the candidates share the normals
    return {"bytes": 8 * case["candidates"], "flops": case["n"] * 252 * (2 * NORMAL + prices * HESTON_STEP)}


# --- the same in 64 bits --------------------------------------------------------------------------

U32 = 0xFFFFFFFF


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _normals(seed, block, paths):
    """The four normals of each Philox block: [4, *shape of block and paths], 64-bit."""
    c = [block + 0 * paths, paths + 0 * block, torch.zeros_like(paths + block), torch.zeros_like(paths + block)]
    k0, k1 = seed & U32, (seed >> 32) & U32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # the low 64 bits are the product's
        c = [((p1 >> 32) & U32) ^ c[1] ^ k0, p1 & U32, ((p0 >> 32) & U32) ^ c[3] ^ k1, p0 & U32]
        k0, k1 = (k0 + 0x9E3779B9) & U32, (k1 + 0xBB67AE85) & U32
    out = []
    for a, b in ((c[0], c[1]), (c[2], c[3])):
        r = torch.sqrt(-2.0 * torch.log((a.double() + 0.5) * 2.0 ** -32))
        th = 2.0 * math.pi * ((b.double() + 0.5) * 2.0 ** -32)
        out += [r * torch.cos(th), r * torch.sin(th)]
    return out


def _stream(seed, n, draws, first=0):
    """The path normals draw by draw (tensors of n), some blocks at a time."""
    paths = torch.arange(first, first + n, dtype=torch.int64, device=_device())[None, :]
    blocks, group = (draws + 3) // 4, max(1, (1 << 21) // n)
    for b0 in range(0, blocks, group):
        blk = torch.arange(b0, min(blocks, b0 + group), dtype=torch.int64, device=_device())[:, None]
        z = _normals(seed, blk, paths)
        for i in range(blk.shape[0]):
            for j in range(4):
                if 4 * (b0 + i) + j < draws:
                    yield z[j][i]


def _grid(dates, spy, fine):
    pts = [0.0] + sorted(dates) + [max(dates)]
    if fine:
        n = math.ceil(max(dates) * spy)
        pts += [max(dates) * k / n for k in range(1, n + 1)]
    out = []
    for x in sorted(pts):
        if not out or abs(x - out[-1]) >= 1e-12:
            out.append(x)
    return out


def _gbm(seed, n, grid, s0, sigma, rate):
    """(dt, normal, log-spot over s0) of every step."""
    y = torch.zeros(n, dtype=torch.float64, device=_device())
    z = _stream(seed, n, len(grid) - 1)
    for k in range(1, len(grid)):
        dt, zz = grid[k] - grid[k - 1], next(z)
        y = y + ((rate - 0.5 * sigma * sigma) * dt + sigma * math.sqrt(dt) * zz)
        yield dt, zz, y


def _heston_paths(seed, n, grid, p, rate, truncate=True):
    y = torch.zeros(n, dtype=torch.float64, device=_device())
    v = torch.full_like(y, p["v0"])
    rp = math.sqrt(max(0.0, 1.0 - p["rho"] ** 2))
    z = _stream(seed, n, 2 * (len(grid) - 1))
    for k in range(1, len(grid)):
        dt = grid[k] - grid[k - 1]
        sq, z1, z2, vp = math.sqrt(dt), next(z), next(z), v.clamp(min=0.0)
        root = vp.sqrt()
        y = y + ((rate - 0.5 * vp) * dt + root * z1 * sq)
        v = v + p["kappa"] * (p["theta"] - vp) * dt + p["sigma_v"] * root * (p["rho"] * z1 + rp * z2) * sq
        if not truncate:
            v = v.clamp(min=0.0)
        yield y


def _values(b, spy, n, s0, sigma, rate, seed):
    """Discounted values of a product's paths under GBM."""
    t, k = b["maturity"], b["strike"]
    grid = _grid([t], spy, b["product"] != "european")
    dev = _device()
    total = torch.full((n,), s0, dtype=torch.float64, device=dev)
    hit = torch.zeros(n, dtype=torch.bool, device=dev)
    if b["product"] == "up_and_out":
        hit |= s0 >= b["barrier"]
    elif b["product"] == "knock_in":
        hit |= s0 <= b["barrier"]
    for _, _, y in _gbm(seed, n, grid, s0, sigma, rate):
        if b["product"] == "asian":
            total += s0 * torch.exp(y)
        elif b["product"] == "up_and_out":
            hit |= y >= math.log(b["barrier"] / s0)
        elif b["product"] == "knock_in":
            hit |= y <= math.log(b["barrier"] / s0)
    s = s0 * torch.exp(y)
    if b["product"] == "asian":
        v = (total / len(grid) - k).clamp(min=0.0)
    elif b["product"] == "knock_in":
        v = torch.where(hit, (k - s).clamp(min=0.0), 0.0)
    else:
        v = (s - k).clamp(min=0.0)
        if b["product"] == "up_and_out":
            v = torch.where(hit, 0.0, v)
    return v * math.exp(-rate * t)


def _summary(v):
    n = v.numel()
    std = float(v.std()) if n > 1 else 0.0
    return {"price": float(v.mean()), "sample_std": std, "std_error": std / math.sqrt(n)}


def _exact_gbm_adjoint(case, seed):
    """Pathwise derivatives in s0, sigma and r; a knock-out survives with a logistic weight per step."""
    p, n, t, rate = _market(case, seed), case["n"], case["maturity"], case["rate"]
    s0, sigma = p["s0"], p["sigma"]
    grid = _grid([t], case["spy"], True)
    dev = _device()
    zero = torch.zeros(n, dtype=torch.float64, device=dev)
    dsig, lw, dlw, total, dtotal, now = zero, zero.clone(), [zero.clone() for _ in range(3)], zero + s0, \
        [zero + 1.0, zero.clone(), zero.clone()], 0.0
    width = 0.5 * sigma * math.sqrt(t / (len(grid) - 1))
    knock = case["product"] == "up_and_out"
    b = math.log(case["barrier"] / s0)
    if knock:
        lw = lw - math.log1p(math.exp(-b / width))
        dlw[0] = dlw[0] - (1.0 - 1.0 / (1.0 + math.exp(-b / width))) / width / s0
    for dt, z, y in _gbm(p["seed"], n, grid, s0, sigma, rate):
        now += dt
        dsig = dsig - sigma * dt + math.sqrt(dt) * z
        dy = (1.0 / s0, dsig, now)  # of the log of the spot
        if knock:
            x = (y - b) / width
            lw = lw - torch.nn.functional.softplus(x, threshold=1e9)
            m = torch.sigmoid(x) / width
            dlw = [d - m * e for d, e in zip(dlw, dy)]
        else:
            s = s0 * torch.exp(y)
            total = total + s
            dtotal = [d + s * e for d, e in zip(dtotal, dy)]
    df = math.exp(-rate * t)
    if knock:
        s, w = s0 * torch.exp(y), torch.exp(lw)
        pay, on = (s - case["strike"]).clamp(min=0.0), (s > case["strike"]).double()
        pv = df * w * pay
        ds = [df * w * on * s * e + pv * d for e, d in zip(dy, dlw)]
    else:
        a = total / len(grid)
        pv, on = df * (a - case["strike"]).clamp(min=0.0), (a > case["strike"]).double()
        ds = [df * on * d / len(grid) for d in dtotal]
    ds[2] = ds[2] - t * pv
    return _sens(pv, dict(zip(SENS["gbm"], ds)))


def _exact_heston_adjoint(case, seed):
    p, n, t, rate = _heston_market(seed, case["s0"]), case["n"], case["maturity"], case["rate"]
    grid = _grid([t], case["spy"], True)
    dev = _device()
    y = torch.zeros(n, dtype=torch.float64, device=dev)
    v = torch.full_like(y, p["v0"])
    kap, th, sv, rho = p["kappa"], p["theta"], p["sigma_v"], p["rho"]
    rp = math.sqrt(1.0 - rho * rho)
    names = ("v0", "kappa", "theta", "sigma_v", "rho")
    dy = {q: torch.zeros_like(y) for q in names}
    dv = {q: torch.zeros_like(y) for q in names}
    dv["v0"] += 1.0
    z = _stream(p["seed"], n, 2 * (len(grid) - 1))
    for k in range(1, len(grid)):
        dt = grid[k] - grid[k - 1]
        sq, z1, z2 = math.sqrt(dt), next(z), next(z)
        vp, m = v.clamp(min=0.0), (v > 0.0).double()
        root = vp.sqrt()
        slope = torch.where(root > 0.0, 0.5 / root, 0.0)
        mix = rho * z1 + rp * z2
        ydv, vdv = (-0.5 * dt + z1 * sq * slope) * m, 1.0 + (-kap * dt + sv * mix * sq * slope) * m
        own = {"v0": 0.0, "kappa": (th - vp) * dt, "theta": kap * dt, "sigma_v": root * mix * sq,
               "rho": sv * root * (z1 - rho / rp * z2) * sq}
        y = y + ((rate - 0.5 * vp) * dt + root * z1 * sq)
        v = v + kap * (th - vp) * dt + sv * root * mix * sq
        for q in names:
            dy[q] = dy[q] + ydv * dv[q]
            dv[q] = vdv * dv[q] + own[q]
    s, df = p["s0"] * torch.exp(y), math.exp(-rate * t)
    pv, g = df * (s - case["strike"]).clamp(min=0.0), df * s * (s > case["strike"]).double()
    ds = {"s0": g / p["s0"], "r": t * (g - pv), **{q: g * dy[q] for q in names}}
    return _sens(pv, {q: ds[q] for q in SENS["heston"]})


def _sens(pv, ds):
    n = pv.numel()
    out = {"price": float(pv.mean()), "price_se": float(pv.std()) / math.sqrt(n)}
    for q, d in ds.items():
        out["d_" + q], out["se_" + q] = float(d.mean()), float(d.std()) / math.sqrt(n)
    return out


def _exact_greeks(case, seed):
    p, r = _market(case, seed), case["rate"]
    hs, hv, hr = 1e-2 * p["s0"], 1e-2 * p["sigma"], 1e-2 * r
    val = lambda s=0.0, v=0.0, q=0.0: _values(case, case["spy"], case["n"], p["s0"] + s, p["sigma"] + v,  # noqa: E731
                                              r + q, p["seed"])
    base, up, dn = val(), val(s=hs), val(s=-hs)
    est = {"price": base, "delta": (up - dn) / (2 * hs), "gamma": (up - 2.0 * base + dn) / (hs * hs),
           "vega": (val(v=hv) - val(v=-hv)) / (2 * hv), "rho": (val(q=hr) - val(q=-hr)) / (2 * hr)}
    out = {k: float(e.mean()) for k, e in est.items()}
    out.update({k + "_se": float(e.std()) / math.sqrt(case["n"]) for k, e in est.items()})
    return out


def _exact_american(case, seed):
    p, n, k, m = _market(case, seed), case["n"], case["strike"], case["n_basis"]
    grid = [0.0] + _dates(case)
    spots = [p["s0"] * torch.exp(y) for _, _, y in _gbm(p["seed"], n, grid, p["s0"], p["sigma"], case["rate"])]

    def basis(s):
        x = s / p["s0"]
        if case["basis"] == "monomial":
            return [x ** j for j in range(m)]
        f = [torch.ones_like(x), 1.0 - x]
        for j in range(1, m - 1):
            f.append(((2 * j + 1 - x) * f[j] - j * f[j - 1]) / (j + 1))
        w = torch.exp(-0.5 * x)
        return [w * g for g in f[:m]]

    value = (k - spots[-1]).clamp(min=0.0)
    for d in range(len(spots) - 2, -1, -1):
        value = value * math.exp(-case["rate"] * (grid[d + 2] - grid[d + 1]))
        pay = (k - spots[d]).clamp(min=0.0)
        itm = pay > 0.0
        if int(itm.sum()) >= m:
            a = basis(spots[d][itm])
            gram = [[float((f * g).sum()) for g in a] for f in a]  # sums of products: no library's choice of GEMM
            coef = np.linalg.solve(np.array(gram), np.array([float((f * value[itm]).sum()) for f in a]))
            exercise = torch.zeros_like(itm)
            exercise[itm] = pay[itm] > sum(float(c) * f for c, f in zip(coef, a))
            value = torch.where(exercise, pay, value)
    return _summary(value * math.exp(-case["rate"] * grid[1]))


def _exact_basket(case, seed):
    p, n, f = _basket(case, seed), case["n"], case["factors"]
    grid = _grid([case["maturity"]], case["spy"], True)
    low = torch.linalg.cholesky(torch.tensor(p["corr"], dtype=torch.float64)).tolist()
    dev = _device()
    y = [torch.zeros(n, dtype=torch.float64, device=dev) for _ in range(f)]
    z = _stream(p["seed"], n, f * (len(grid) - 1))
    level = sum(p["s0"]) / f
    hit = torch.full((n,), level >= case["barrier"], device=dev)
    for k in range(1, len(grid)):
        dt, zz = grid[k] - grid[k - 1], [next(z) for _ in range(f)]
        for i in range(f):
            w, v = sum(low[i][j] * zz[j] for j in range(i + 1)), p["sigma"][i]
            y[i] = y[i] + ((p["rate"] - 0.5 * v * v) * dt + v * math.sqrt(dt) * w)
        level = sum(s * torch.exp(x) for s, x in zip(p["s0"], y)) / f
        hit |= level >= case["barrier"]
    v = torch.where(hit, 0.0, (level - case["strike"]).clamp(min=0.0))
    return _summary(v * math.exp(-p["rate"] * case["maturity"]))


def _exact_calibration(case, seed):
    p, n = _calibration(case, seed), case["n"]
    grid = _grid([p["maturity"]], 252, True)
    col = lambda i: torch.tensor([c[i] for c in p["population"]], dtype=torch.float64, device=_device())[:, None]  # noqa: E731
    v0, kap, th, sv, rho = (col(i) for i in range(5))
    rp = (1.0 - rho * rho).clamp(min=0.0).sqrt()
    y = torch.zeros(len(p["population"]), n, dtype=torch.float64, device=_device())
    v = v0 + 0.0 * y
    z = _stream(42, n, 2 * (len(grid) - 1))  # every price of a calibration draws from seed 42
    for k in range(1, len(grid)):
        dt = grid[k] - grid[k - 1]
        sq, z1, z2, root = math.sqrt(dt), next(z)[None], next(z)[None], v.sqrt()
        y = y + ((p["rate"] - 0.5 * v) * dt + root * z1 * sq)
        v = (v + kap * (th - v) * dt + sv * root * (rho * z1 + rp * z2) * sq).clamp(min=0.0)
    df, obj = math.exp(-p["rate"] * p["maturity"]), 0.0
    for s, quote in p["quotes"]:
        price = df * (s * torch.exp(y) - p["strike"]).clamp(min=0.0).mean(1)
        obj = obj + (price - quote) ** 2
    return (obj / len(p["quotes"])).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "price":
        if case["model"] == "heston":
            p, t = _heston_market(seed, case["s0"]), case["maturity"]
            for y in _heston_paths(p["seed"], case["n"], _grid([t], case["spy"], True), p, case["rate"]):
                pass
            v = math.exp(-case["rate"] * t) * (p["s0"] * torch.exp(y) - case["strike"]).clamp(min=0.0)
        else:
            p = _market(case, seed)
            v = _values(case, case["spy"], case["n"], p["s0"], p["sigma"], case["rate"], p["seed"])
        out = _summary(v)
        return {k: np.float64(x) for k, x in out.items()} if case["precision"] == "fp64" else out
    if kind == "heston_book":
        p, ladder = _heston_market(seed), _heston_ladder(case)
        grid = _grid([t for _, t in ladder], case["spy"], True)
        spot = {}
        for k, y in enumerate(_heston_paths(p["seed"], case["n"], grid, p, 0.05), 1):
            for t in {t for _, t in ladder}:
                if abs(grid[k] - t) < 1e-12:
                    spot[t] = p["s0"] * torch.exp(y)
        rows = [_summary(math.exp(-0.05 * t) * (spot[t] - k).clamp(min=0.0)) for k, t in ladder]
    elif kind == "book":
        rows = [_summary(_values(b, case["spy"], b["n"], b["s0"], b["sigma"], b["rate"], b["seed"]))
                for b in _book(case, seed)]
    elif kind == "greeks":
        return _exact_greeks(case, seed)
    elif kind == "adjoint":
        return _exact_heston_adjoint(case, seed) if case["model"] == "heston" else _exact_gbm_adjoint(case, seed)
    elif kind == "american":
        return _exact_american(case, seed)
    elif kind == "basket":
        return _exact_basket(case, seed)
    else:
        return _exact_calibration(case, seed)
    return {q: np.array([r[q] for r in rows]) for q in ("price", "sample_std", "std_error")}
