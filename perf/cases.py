"""Timed cases of the pricing engine: what a desk has it do, from one small price to a book.

A case is one call of a public entry point (a fixed-size pass, a level pair, a sensitivity run, an adaptive
driver, a book) on a product drawn from a seed around the repository's own workloads: the arithmetic Asian under
GBM (256 steps, 32 replicas), the Heston lookback under MLQMC, the 64 x 32 local-vol surface with node vegas, the
heterogeneous basket book, the reference examples' short European runs.

Results are returned as FP32: every path is priced in FP32 and only the sums over paths are doubles, so the
digits beyond FP32 are rounding noise of the paths.  Sample sizes of the drivers that size their runs from a variance
estimate (MLQMC, MLMC, the book) are not returned: the last bit of the estimate moves a ceil().  Knock-out
barriers are left to the tests: one FP32 knock-out flip moves a replica's sum by a whole path.

exact() prices the same points in FP64 with torch alone: JoeKuo6 direction numbers, the Hong-Hickernell
scramble, u = (float(x) + 1) 2^-32 as the stream defines it, Philox4x32-10 with Box-Muller, and the models' Euler
steps.  Sensitivities come from autograd.
"""
import functools
import importlib
import math
import random

import numpy as np
import torch

eng = importlib.import_module("financial-derivatives-montecarlo_b200")

NOISE = {"raw": eng.RAW, "bridge": eng.BB, "pca": eng.PCA}


def listed():
    return [
        # one cheap price on request: latency of a synchronous call, a few launches, almost no work
        dict(name="quote_european", kind="qmc", model="gbm", payoff="european", steps=16, noise="raw", R=8,
             points=1000, offset=0, device=False),
        # plain Monte Carlo of a short European (the reference's first example)
        dict(name="mc_european", kind="mc", model="gbm", payoff="european", steps=64, points=1000000),
        # the headline pass: arithmetic Asian, 32 replicas, everything resident on the device
        dict(name="asian_raw_large", kind="qmc", model="gbm", payoff="asian", steps=256, noise="raw", R=32,
             points=1 << 20, offset=0, device=True),
        # the same product in the two other orderings, at a doubling of ordinary size
        dict(name="asian_bridge", kind="qmc", model="gbm", payoff="asian", steps=256, noise="bridge", R=32,
             points=131071, offset=131072, device=False),
        dict(name="asian_pca", kind="qmc", model="gbm", payoff="asian", steps=256, noise="pca", R=32,
             points=1 << 17, offset=0, device=False),
        # ragged sizes: steps and points that fill no tile, from an odd point on
        dict(name="dupire_ragged", kind="qmc", model="dupire", payoff="european", steps=100, noise="raw", R=16,
             points=100003, offset=4097, device=False),
        # a fine / coarse pair of the Heston MLQMC, the unit of its deep levels
        dict(name="heston_level", kind="level", model="heston", payoff="lookback", steps=256, M=4, sobol=True, R=32,
             points=1 << 15, offset=0),
        # a weekly-monitored basket of correlated assets in one pass
        dict(name="basket_weekly", kind="qmc", model="basket", assets=5, payoff="basket", steps=52, noise="raw", R=16,
             points=1 << 16, offset=0, device=False),
        # all sensitivities of a local-vol Asian, node vegas among them
        dict(name="localvol_greeks", kind="greeks", model="localvol", payoff="asian", steps=512, R=16, points=60000),
        # the adaptive drivers: RQMC by doubling, MLQMC by levels, a book of baskets
        dict(name="asian_driver", kind="qmc_driver", model="gbm", payoff="asian", steps=256, noise="raw", R=32,
             start=1 << 14, eps=1e-3),
        dict(name="heston_mlqmc", kind="mlqmc", model="heston", payoff="lookback", eps=1e-3, M=4, n0=4, R=32),
        dict(name="basket_book", kind="book", options=48, eps=2.5e-3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["qmc"] * 6 + ["mc", "level", "level", "greeks", "qmc_driver", "mlqmc", "book"])
    R = rng.choice([8, 16, 32])
    points = _log_int(rng, 1 << 9, 1 << 19)
    payoff = rng.choice(["european", "asian", "geometric", "lookback"])
    offset = rng.choice([0, points, rng.randrange(1, 1 << 16)])
    if kind == "qmc":
        model = rng.choice(["gbm", "gbm", "heston", "dupire", "localvol", "basket"])
        case = dict(kind=kind, model=model, payoff=payoff, steps=_log_int(rng, 1, 512), noise="raw", R=R,
                    points=points, offset=offset, device=rng.random() < 0.3)
        if model == "basket":
            case.update(payoff="basket", assets=rng.randrange(2, 17), steps=_log_int(rng, 1, 64))
        elif model in ("gbm", "dupire", "localvol"):
            case["noise"] = rng.choice(["raw", "raw", "bridge", "pca"])
            if case["noise"] == "bridge":
                case["steps"] = 1 << rng.randrange(2, 10)
            elif case["noise"] == "pca":
                case["steps"] = rng.choice([8, 32, 64, 128, 256])
        per = case["steps"] * case.get("assets", 2 if model == "heston" else 1)
        case["points"] = max(256, min(points, (1 << 31) // (R * per)))
        return case
    if kind == "mc":
        return dict(kind=kind, model=rng.choice(["gbm", "heston", "dupire"]), payoff=payoff,
                    steps=_log_int(rng, 2, 256), points=_log_int(rng, 1 << 12, 1 << 22))
    if kind == "level":
        M = rng.choice([2, 4])
        model = rng.choice(["gbm", "heston", "dupire"])
        steps = M ** rng.randrange(1, 11 if M == 2 else 6)
        return dict(kind=kind, model=model, payoff=payoff, steps=steps, M=M, sobol=rng.random() < 0.7, R=R,
                    points=max(256, min(points, (1 << 30) // (R * steps))), offset=offset)
    if kind == "greeks":
        model = rng.choice(["gbm", "localvol", "heston"])
        return dict(kind=kind, model=model, payoff=rng.choice(["european", "asian", "lookback"]),
                    steps=32 * rng.randrange(1, 17), R=rng.choice([8, 16]), points=_log_int(rng, 1000, 50000))
    if kind == "qmc_driver":
        return dict(kind=kind, model=rng.choice(["gbm", "dupire"]), payoff=rng.choice(["european", "asian"]),
                    steps=_log_int(rng, 8, 256), noise="raw", R=32, start=1 << rng.randrange(10, 15),
                    eps=2e-3 * math.exp(rng.uniform(0.0, math.log(10.0))))
    if kind == "mlqmc":
        return dict(kind=kind, model=rng.choice(["gbm", "heston"]), payoff=rng.choice(["european", "lookback"]),
                    eps=2e-3 * math.exp(rng.uniform(0.0, math.log(10.0))), M=rng.choice([2, 4]), n0=4, R=32)
    return dict(kind=kind, options=rng.randrange(4, 49), eps=2.5e-3 * math.exp(rng.uniform(0.0, math.log(5.0))))


# ---------------------------------------------------------------- inputs

def _inputs(case, seed):
    """The product's numbers, from the seed alone."""
    g = random.Random("%s/%s/%d" % (case.get("model"), case.get("payoff"), seed))
    q = dict(S0=g.uniform(90.0, 110.0), mu=g.uniform(0.01, 0.05), T=g.uniform(0.75, 1.25), sigma=g.uniform(0.15, 0.3),
             kappa=g.uniform(1.5, 2.5), theta=g.uniform(0.03, 0.06), xi=g.uniform(0.2, 0.4), rho=g.uniform(-0.8, -0.5),
             v0=g.uniform(0.03, 0.06), alpha=g.uniform(0.2, 0.6), beta=g.uniform(0.7, 0.9),
             salt=g.randrange(1, 1 << 30))
    q["K"] = q["S0"] * g.uniform(0.9, 1.1)
    if case.get("model") == "localvol":
        q["T"] = 2.0
        q["Kx"], q["tx"], q["grid"] = eng.config4_surface(seed % 100000)
    if case.get("model") == "basket":
        n, r = case["assets"], np.random.default_rng(seed)
        A = r.normal(size=(n, n))
        C = A @ A.T + 0.5 * np.eye(n)
        C /= np.sqrt(np.outer(np.diag(C), np.diag(C)))
        q["S"], q["sig"], q["w"] = 100.0 * r.uniform(0.8, 1.2, n), r.uniform(0.1, 0.5, n), r.dirichlet(np.ones(n))
        q["L"], q["K"] = np.linalg.cholesky(C), float(np.dot(q["w"], q["S"]) * g.uniform(0.9, 1.1))
    return q


def _model(case, q):
    kind = case["model"]
    if kind == "gbm":
        return eng.gbm(q["S0"], q["mu"], q["sigma"], q["T"])
    if kind == "heston":
        return eng.heston(q["S0"], q["mu"], q["kappa"], q["theta"], q["xi"], q["rho"], q["v0"], q["T"])
    if kind == "dupire":
        return eng.dupire(q["S0"], q["mu"], q["sigma"], q["alpha"], q["beta"], q["T"])
    if kind == "localvol":
        return eng.localvol_grid(q["Kx"], q["tx"], q["grid"], q["S0"], q["mu"], q["T"])
    return eng.basket_gbm(q["S"], q["sig"], L=q["L"], weights=q["w"], mu=q["mu"], T=q["T"])


def _payoff(case, q):
    kind = case["payoff"]
    if kind == "european":
        return eng.european(q["K"], q["mu"], q["T"])
    if kind == "basket":
        return eng.basket(q["K"], q["mu"], q["T"], case["assets"])
    return {"asian": lambda: eng.asian(q["K"]), "geometric": lambda: eng.geom_asian(q["K"]),
            "lookback": lambda: eng.lookback(q["sigma"])}[kind]()


def _flags(case):
    return eng.FLAG_HESTON_MILSTEIN if case.get("model") == "heston" and case["kind"] != "mc" else 0


@functools.lru_cache(maxsize=None)
def _pricing_stream():
    """The one stream of a program that leaves its results on the device."""
    return torch.cuda.Stream()


def prepare(case, seed):
    """Model and payoff structs, the ordering's handle, and for a device pass the result buffer."""
    s = dict(case=case)
    if case["kind"] == "book":
        s["options"] = eng.config5_book(case["options"], seed=seed % (1 << 31))
        for o in s["options"]:
            o.eps = case["eps"]
            o.max_L = min(o.max_L, 7)
        return s
    q = _inputs(case, seed)
    s.update(q=q, model=_model(case, q), payoff=_payoff(case, q), flags=_flags(case), salt=q["salt"])
    if case.get("noise") == "bridge":
        s["bb"] = eng.bb_create(case["steps"], q["T"])
    if case.get("noise") == "pca":
        s["pca"] = eng.pca_create(case["steps"], q["T"])
    if case.get("device"):
        with torch.cuda.stream(_pricing_stream()):
            s["sums"] = torch.zeros(case["R"], 2, dtype=torch.float64, device="cuda")
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "book":
        res, _ = eng.book_price(s["options"])
        delta = np.zeros((len(res), 16), np.float32)
        for row, r in zip(delta, res):
            row[:r["delta"].size] = r["delta"]
        return {"price": np.array([[r["price"], r["std_error"]] for r in res], np.float32), "delta": delta}
    m, p = s["model"], s["payoff"]
    if kind == "qmc":
        where = dict(noise=NOISE[c["noise"]], bb=s.get("bb"), pca=s.get("pca"), salt_base=s["salt"], R=c["R"],
                     offset=c["offset"], n_points=c["points"], flags=s["flags"])
        if c["device"]:
            with torch.cuda.stream(_pricing_stream()):
                eng.qmc_pass_device(m, p, c["steps"], s["sums"].data_ptr(), _pricing_stream().cuda_stream, **where)
                return (s["sums"] / c["points"]).float()
        return (eng.qmc_pass(m, p, c["steps"], **where) / c["points"]).astype(np.float32)
    if kind == "mc":
        return np.array(eng.run_mc_fixed(m, p, c["steps"], c["points"], s["salt"]), np.float32)
    if kind == "level":
        sums = eng.level_pass(m, p, c["steps"], c["M"], use_sobol=c["sobol"], seed=s["salt"], salt_base=s["salt"],
                              R=c["R"], offset=c["offset"], n_points=c["points"], flags=s["flags"])
        return (sums / c["points"]).astype(np.float32)
    if kind == "greeks":
        g, nodes = eng.adjoint(m, p, c["steps"], salt_base=s["salt"], R=c["R"], n_points=c["points"], flags=s["flags"])
        out = {"greeks": np.array([g[k] for k in ("price", "delta", "rho", "vega", "price_se", "delta_se", "rho_se",
                                                  "vega_se")], np.float32)}
        if nodes is not None:
            out["nodes"] = nodes.astype(np.float32)
        return out
    if kind == "qmc_driver":
        cfg = eng.qmc_cfg(R=c["R"], N0_per_replica=c["start"], salt_base=s["salt"], max_doublings=8)
        r = eng.run_qmc(m, p, c["eps"], c["steps"], cfg)
        return {"price": np.array([r["price"], r["std_error"]], np.float32), "samples": r["n_samples"]}
    ml = eng.mlmc_cfg(M=c["M"], n0_steps=c["n0"], max_L=8 if c["M"] == 2 else 6, flags=s["flags"])
    r = eng.run_mlqmc(m, p, c["eps"], ml, eng.qmc_cfg(R=c["R"], salt_base=s["salt"], flags=s["flags"]))
    return np.array([r["price"], r["std_error"]], np.float32)


def work(case):
    """FP32 operations of one pass: per normal one XOR, two for u and an inverse normal of about ten (or an eighth
    of two Philox blocks and half a Box-Muller pair), per step the model's Euler update and the payoff's running
    term; three sweeps for sensitivities.  The traffic is the direction numbers and the results."""
    kind = case["kind"]
    if kind == "book":      # normals of such an option from the adaptive rule, about 1.6e4 / eps^2
        return {"bytes": 4096.0 * case["options"], "flops": case["options"] * 1.6e4 / case["eps"] ** 2 * 20.0}
    step = {"gbm": 5.0, "heston": 18.0, "dupire": 11.0, "localvol": 19.0, "basket": 5.0}[case["model"]]
    width = case.get("assets", 2 if case["model"] == "heston" else 1)
    if case["model"] == "basket":
        step = width * (4.0 + width)
    if kind == "mlqmc":     # path-steps of such a run, about 4e4 / eps^2
        return {"bytes": 1e6, "flops": 4e4 / case["eps"] ** 2 * (13.0 * width + step)}
    steps = case["steps"]
    paths = case.get("R", 1) * case.get("points", case.get("start", 0))
    if kind == "qmc_driver":    # doublings to a standard error of eps / sqrt(2): about 6e6 points at 1e-3
        paths = max(paths, 6e6 * (1e-3 / case["eps"]))
    per = 13.0 * width + step
    if kind == "level":
        per += step / case["M"]
    if kind == "greeks":
        per += 2.0 * step
    return {"bytes": 4.0 * 33 * steps * width * case.get("R", 1) + 64.0, "flops": paths * steps * per}


# ---------------------------------------------------------------- the same points in FP64

_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_M32 = 0xFFFFFFFF


def _mix(x):
    x = (x + 0x9E3779B9) & _M32
    x = ((x ^ (x >> 16)) * 0x21F0AAAD) & _M32
    x = ((x ^ (x >> 15)) * 0x735A2D97) & _M32
    return x ^ (x >> 15)


class _Sobol:
    """Scrambled Sobol normals of R replicas, dimension by dimension, for an aligned block of points."""

    def __init__(self, salt, R, D):
        v = torch.quasirandom.SobolEngine(D, scramble=False).sobolstate.to(_DEV).long() << 2     # [D, 30]
        base = torch.tensor([_mix((salt + r) & _M32) for r in range(R)], device=_DEV)[:, None] ^ torch.arange(D, device=_DEV)
        self.words = torch.zeros(R, D, 30, dtype=torch.int64, device=_DEV)
        for k in range(32):
            row = (1 << (31 - k)) | (_mix(base ^ k) & ((_M32 << (32 - k)) & _M32))
            b = row[:, :, None] & v
            for s in (16, 8, 4, 2, 1):
                b = b ^ (b >> s)
            self.words |= (b & 1) << (31 - k)
        self.shift = _mix(base ^ 0xA5A5A5A5)
        self.lo = self._of(torch.arange(1024, device=_DEV))

    def _of(self, n):
        g = n ^ (n >> 1)
        x = torch.zeros(self.words.shape[0], self.words.shape[1], n.numel(), dtype=torch.int64, device=_DEV)
        for k in range(30):
            bit = (g >> k) & 1
            if bool(bit.any()):
                x ^= self.words[:, :, k, None] * bit
        return x

    def block(self, first, count):
        self.hi = self._of(torch.arange(first, first + count, 1024, device=_DEV)) ^ self.shift[:, :, None]

    def normal(self, d):
        x = (self.hi[:, d, :, None] ^ self.lo[:, d, None, :]).flatten(1)
        u = x.float() * 2.0 ** -32 + 2.0 ** -32
        return torch.special.ndtri(u.clamp(max=1.0 - 2.0 ** -24).double())


class _Philox:
    """Philox4x32-10 with Box-Muller: four normals of a path per counter block."""

    def __init__(self, seed, streams):
        self.seed, self.streams = seed, torch.tensor(streams, device=_DEV)[:, None]

    def block(self, first, count):
        self.path, self.at = torch.arange(first, first + count, device=_DEV)[None, :], -1

    def normal(self, d):
        if d // 4 != self.at:
            self.at = d // 4
            one = torch.ones_like(self.path * self.streams)
            c = [one * self.at, one * (self.path & _M32), one * (self.path >> 32), one * self.streams]
            k0, k1 = self.seed, 0x6D637121
            for _ in range(10):
                p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
                c = [((p1 >> 32) & _M32) ^ c[1] ^ k0, p1 & _M32, ((p0 >> 32) & _M32) ^ c[3] ^ k1, p0 & _M32]
                k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
            u = [((x >> 8).float() + 0.5) * 2.0 ** -24 for x in c]
            self.z = []
            for a, b in ((u[0], u[1]), (u[2], u[3])):
                rr, t = torch.sqrt(-2.0 * torch.log(a.double())), 2.0 * math.pi * b.double()
                self.z += [rr * torch.sin(t), rr * torch.cos(t)]
        return self.z[d % 4]


def _increments(case, T, gen):
    """A function of the step: its scaled increments, one tensor [R, points] per factor."""
    n, width = case["steps"], case.get("assets", 2 if case["model"] == "heston" else 1)
    h, noise = T / n, case.get("noise", "raw")
    if noise == "raw":
        return lambda k: [gen.normal(k * width + f) * math.sqrt(h) for f in range(width)]
    z = [gen.normal(d) for d in range(n)]
    if noise == "bridge":
        W = {0: torch.zeros_like(z[0]), n: math.sqrt(T) * z[0]}
        d, stride = 1, n
        while stride > 1:
            for a in range(0, n, stride):
                W[a + stride // 2] = 0.5 * (W[a] + W[a + stride]) + math.sqrt(0.25 * stride * h) * z[d]
                d += 1
            stride //= 2
        return lambda k: [W[k + 1] - W[k]]
    j = torch.arange(1, n + 1, device=_DEV, dtype=torch.float64)
    lam = h / (4.0 * torch.sin((2 * j - 1) * math.pi / (2 * (2 * n + 1))) ** 2)
    V = 2.0 / math.sqrt(2 * n + 1) * torch.sin(j[:, None] * (2 * j - 1) * math.pi / (2 * n + 1)) * torch.sqrt(lam)
    M = torch.cat([V[:1], V[1:] - V[:-1]])
    dW = torch.stack(z, -1) @ M.T
    return lambda k: [dW[..., k]]


class _Leg:
    """One discretisation of the product's paths; S0, rate, vol (and the grid) may carry gradients."""

    def __init__(self, case, q, par, n, like):
        self.c, self.q, self.par, self.n, self.h, self.k = case, q, par, n, q["T"] / n, 0
        self.S = par["S0"] + torch.zeros_like(like)
        self.V = (par["vol"] if case["model"] == "heston" else 0.0) + torch.zeros_like(like)
        self.run = self.S if case["payoff"] == "lookback" else torch.zeros_like(like)
        if case["model"] == "basket":
            self.S = [torch.full_like(like, float(x)) for x in q["S"]]

    def step(self, dw, milstein):
        c, q, p, S, h = self.c["model"], self.q, self.par, self.S, self.h
        if c == "basket":
            self.S = [S[a] + S[a] * (p["rate"] * h + q["sig"][a] * sum(q["L"][a][b] * dw[b] for b in range(a + 1)))
                      for a in range(len(S))]
            return
        if c == "gbm":
            vol = p["vol"]
        elif c == "dupire":
            vol = p["vol"] * math.exp(-q["alpha"] * self.k * h) * (S / p["S0"]) ** (q["beta"] - 1.0)
        elif c == "localvol":
            nt, nK = q["grid"].shape
            dK, dt = q["Kx"][1] - q["Kx"][0], q["tx"][1] - q["tx"][0]
            y = min(max((self.k * h - q["tx"][0]) / dt, 0.0), nt - 1.0)
            j = min(int(y), nt - 2)
            x = ((S - q["Kx"][0]) / dK).clamp(0.0, nK - 1.0)
            i = x.detach().long().clamp(max=nK - 2)
            row = (1 - (y - j)) * p["grid"][:, j] + (y - j) * p["grid"][:, j + 1]
            lo = row.gather(1, i)
            vol = lo + (x - i) * (row.gather(1, i + 1) - lo)
        else:
            Vp = self.V.clamp(min=0.0)
            vol = torch.where(Vp > 0, torch.sqrt(torch.where(Vp > 0, Vp, torch.ones_like(Vp))), torch.zeros_like(Vp))
            w2 = q["rho"] * dw[0] + math.sqrt(1.0 - q["rho"] ** 2) * dw[1]
            V = q["theta"] + math.exp(-q["kappa"] * h) * (self.V - q["theta"]) + q["xi"] * vol * w2
            self.V = V + 0.25 * q["xi"] ** 2 * (w2 * w2 - h) if milstein else V
        self.S = S = S + S * (p["rate"] * h + vol * dw[0])
        self.k += 1
        pay = self.c["payoff"]
        if pay == "asian":
            self.run = self.run + S
        elif pay == "geometric":
            self.run = self.run + torch.log(S)
        elif pay == "lookback":
            self.run = torch.minimum(self.run, S)

    def payoff(self):
        pay, q = self.c["payoff"], self.q
        if pay == "asian":
            return (self.run / self.n - q["K"]).clamp(min=0.0)
        if pay == "geometric":
            return (torch.exp(self.run / self.n) - q["K"]).clamp(min=0.0)
        if pay == "lookback":
            return self.S - self.run * math.exp(-float(np.float32(0.5826)) * q["sigma"] * math.sqrt(self.h))
        B = sum(float(w) * s for w, s in zip(q["w"], self.S)) if pay == "basket" else self.S
        disc = self.par["disc"](q["T"])
        return (B - q["K"]).clamp(min=0.0) * disc


def _paths(case, q, par, gen, first, count):
    """Payoffs of points first .. first + count - 1: (fine, coarse or None), [R, count]."""
    a = first & ~1023
    b = (first + count + 1023) & ~1023
    gen.block(a, b - a)
    cut = slice(first - a, first - a + count)
    dW, n, M = _increments(case, q["T"], gen), case["steps"], case.get("M", 0)
    mil = bool(_flags(case))
    fine = coarse = None
    for k in range(n):
        dw = [x[:, cut] for x in dW(k)]
        if fine is None:
            fine = _Leg(case, q, par, n, dw[0])
            coarse, acc = (_Leg(case, q, par, n // M, dw[0]) if M else None), None
        fine.step(dw, mil)
        if M:
            acc = dw if acc is None else [x + y for x, y in zip(acc, dw)]
            if (k + 1) % M == 0:
                coarse.step(acc, mil)
                acc = None
    return fine.payoff(), coarse.payoff() if M else None


def _chunks(case, total, offset):
    """Point ranges of a size that fits: 2^23 paths at a time, fewer where whole paths are held."""
    room = 1 << 23
    if case["kind"] == "greeks":
        room = (1 << 28) // (case["steps"] * (3 if case["model"] == "gbm" else 8) // 2)
    elif case.get("noise", "raw") != "raw":
        room = (1 << 30) // case["steps"]
    size = max(1024, room // case.get("R", 1) // 1024 * 1024)
    first = offset
    while first < offset + total:
        last = min(offset + total, (first // size + 1) * size)
        yield first, last - first
        first = last


def _params(case, q, R, grads=False):
    t = lambda x: torch.full((R, 1), x, dtype=torch.float64, device=_DEV, requires_grad=grads)  # noqa: E731
    vol = q["v0"] if case["model"] == "heston" else q["sigma"]
    p = dict(S0=t(q["S0"]), rate=t(q["mu"]), vol=t(vol))
    p["disc"] = lambda T: torch.exp(-p["rate"] * T)
    if case["model"] == "localvol":
        g = torch.tensor(q["grid"], device=_DEV)
        p["grid"] = g.expand(R, *g.shape).clone().requires_grad_(grads)
    return p


def _sums(case, q, gen, R, total, offset):
    """[R, 2] sums of Y, Y^2 (or [R, 4] of dY, dY^2, Yf, Yf^2) over the points."""
    par, out = _params(case, q, R), 0.0
    for first, count in _chunks(case, total, offset):
        yf, yc = _paths(case, q, par, gen, first, count)
        cols = [yf, yf * yf] if yc is None else [yf - yc, (yf - yc) ** 2, yf, yf * yf]
        out = out + torch.stack([x.sum(1) for x in cols], 1)
    return out.cpu().numpy()


def _greeks(case, q):
    R, n = case["R"], case["points"]
    gen = _Sobol(q["salt"], R, case["steps"] * (2 if case["model"] == "heston" else 1))
    par, Y = _params(case, q, R, True), 0.0
    for first, count in _chunks(case, n, 0):
        y, _ = _paths(case, q, par, gen, first, count)
        y.sum().backward()
        Y = Y + y.detach().sum(1)
    g = par.get("grid")
    vega = par["vol"].grad[:, 0] if g is None else g.grad.flatten(1).sum(1)
    per = torch.stack([Y, par["S0"].grad[:, 0], par["rate"].grad[:, 0], vega]) / n
    out = {"greeks": torch.cat([per.mean(1), per.std(1) / math.sqrt(R)]).cpu().numpy()}
    if g is not None:
        out["nodes"] = (g.grad.sum(0) / (R * n)).cpu().numpy()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("book", "mlqmc"):     # their sample sizes follow from their own estimates
        return None
    q = _inputs(case, seed)
    if kind == "greeks":
        return _greeks(case, q)
    with torch.no_grad():
        if kind == "mc":
            n = case["points"]
            s = _sums(case, q, _Philox(q["salt"], [0]), 1, n, 0)[0] / n
            return np.array([s[0], max(0.0, s[1] - s[0] * s[0]) / n])
        R = case["R"]
        if kind == "level" and not case["sobol"]:
            gen = _Philox(q["salt"], [q["salt"] + r for r in range(R)])
        else:
            gen = _Sobol(q["salt"], R, case["steps"] * case.get("assets", 2 if case["model"] == "heston" else 1))
        if kind != "qmc_driver":
            return _sums(case, q, gen, R, case["points"], case["offset"]) / case["points"]
        done, n, total = 0, case["start"], 0.0
        for _ in range(8):
            total, done = total + _sums(case, q, gen, R, n - done, done), n
            means = total[:, 0] / n
            se2 = means.var(ddof=1) / R
            if se2 < case["eps"] ** 2 / 2:
                break
            n *= 2
        return {"price": np.array([means.mean(), math.sqrt(se2)]), "samples": None}
