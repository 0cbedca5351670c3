"""The pricing calls whose speed this repository answers for.

``listed()`` gives the cases, ``draw()`` more of the same ranges.  A case is a
kind of call with its sizes and options; market data and sampling seeds come
from the seed given to ``prepare()``, so the work of a case is the same for
every seed.  ``run()`` is one call of the public Python API
(``montepath_b200.backend.CudaBackend``) on requests the program holds, on the
process-wide device context a program keeps (``montepath_b200.native.backend()``).
``exact()`` states what the call estimates, on the same samples, in 64-bit
torch arithmetic.

Kinds, with the real use each stands for:

terminal    one European call by its terminal distribution: the smallest
            request, where launches and host latency count
gbm_fp64    one GBM option replayed from the reference's random stream in
            FP64: the drop-in call of a user who wants the reference's numbers
exotics     a desk's mixed batch of path-dependent options on the default
            pseudorandom stream, one technique each
structured  the other sample sequences: randomized Halton, Latin hypercube and
            Brownian-bridge Sobol
pair        Heston and Merton calls on scrambled Sobol: the headline workload,
            FP32 paths or FP64
lsm         American (and Bermudan) puts by Longstaff-Schwartz
book        a heterogeneous book of counter-hash contracts in one batch
mlmc        the multilevel arithmetic Asian, with the default allocation
greeks      a Greek report: bump and revalue, pathwise or likelihood ratio
merton      the reference's Merton estimator: the jump-dependent stream replay
"""

from __future__ import annotations

import math
import random
from functools import lru_cache

import numpy as np
import torch

from montepath_b200 import native
from montepath_b200.requests import make_request

BASKET5 = {"spots": [100.0, 95.0, 105.0, 90.0, 110.0], "sigmas": [0.2, 0.25, 0.3, 0.35, 0.4], "corr": 0.3}
HESTON = {"v0": 0.04, "kappa": 2.0, "theta": 0.04, "vol_of_vol": 0.5, "rho": -0.7}
BOOK_KINDS = ("european_call", "arithmetic_asian_call", "up_and_out_call", "basket_call")


# ------------------------------------------------------------------ cases ---
def listed():
    return [
        # the smallest call: a quote of one vanilla option
        dict(name="terminal_10000", kind="terminal", paths=10_000, technique="standard", sampling="pseudorandom"),
        # the repository's first benchmark row, FP64 on the reference's stream
        dict(name="gbm_fp64_20000x64", kind="gbm_fp64", workload="european_call", paths=20_000, steps=64, threads=1,
             technique="standard"),
        # the benchmark harness's path-dependent rows as a desk prices them: in one batch
        dict(name="exotics_100000x64", kind="exotics", paths=100_000, steps=64),
        # the benchmark harness's other sampling methods
        dict(name="structured_100000x64", kind="structured", paths=100_000, steps=64, precision="fp32_path"),
        # the headline workload, and the same models in FP64
        dict(name="pair_1048576x256", kind="pair", paths=1_048_576, steps=256, precision="fp32_path"),
        dict(name="pair_fp64_131072x256", kind="pair", paths=131_072, steps=256, precision="fp64_plain"),
        # the large American put of the benchmark, and a small FP64 batch with a Bermudan
        dict(name="lsm_524288x50", kind="lsm", paths=524_288, steps=50, degree=3, bermudan=False,
             precision="fp32_path"),
        dict(name="lsm_fp64_100000x64", kind="lsm", paths=100_000, steps=64, degree=2, bermudan=True,
             precision="fp64_plain"),
        # a slice of the 4,096-contract book
        dict(name="book_24", kind="book", contracts=24, sizes=42),
        # the default multilevel request
        dict(name="mlmc_4_levels", kind="mlmc", levels=4, base_steps=16, paths=50_000, sampling="counter_hash",
             replicates=1),
        # a risk run: all bump legs of an Asian call
        dict(name="greeks_262144x64", kind="greeks", workload="arithmetic_asian_call", paths=262_144, steps=64,
             sampling="scrambled_sobol", technique="antithetic", precision="fp32_path",
             estimator="bump_and_revalue"),
        # the default Merton request (an odd number of paths)
        dict(name="merton_1000003", kind="merton", paths=1_000_003, threads=1),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    techniques = ("standard", "antithetic", "control_variate")
    kind = rng.choice(("terminal", "gbm_fp64", "exotics", "structured", "pair", "lsm", "book", "mlmc", "greeks",
                       "merton"))
    if kind == "terminal":
        return dict(kind=kind, paths=size(1_000, 4_000_000), technique=rng.choice(techniques),
                    sampling=rng.choice(("pseudorandom", "counter_hash", "scrambled_sobol")))
    if kind == "gbm_fp64":
        return dict(kind=kind, paths=size(1_000, 200_000), steps=size(1, 252), threads=rng.choice((1, 1, 4)),
                    workload=rng.choice(("european_call", "arithmetic_asian_call", "down_and_out_call",
                                         "lookback_call")), technique=rng.choice(techniques))
    if kind == "exotics":
        return dict(kind=kind, paths=size(1_000, 400_000), steps=size(4, 252))
    if kind == "structured":
        precision = rng.choice(("fp32_path", "fp32_path", "fp64_plain"))
        return dict(kind=kind, paths=size(1_000, 130_000), steps=size(2, 128), precision=precision)
    if kind == "pair":
        if rng.random() < 0.5:
            return dict(kind=kind, paths=size(4_000, 1_048_576), steps=rng.randint(16, 256), precision="fp32_path")
        return dict(kind=kind, paths=size(4_000, 131_072), steps=rng.randint(16, 256), precision="fp64_plain")
    if kind == "lsm":
        fp64 = rng.random() < 0.4
        return dict(kind=kind, paths=size(1_000, 150_000 if fp64 else 524_288), steps=rng.randint(8, 64),
                    degree=rng.randint(1, 3), bermudan=fp64, precision="fp64_plain" if fp64 else "fp32_path")
    if kind == "book":
        return dict(kind=kind, contracts=rng.randint(3, 24), sizes=rng.randint(1, 10_000))
    if kind == "mlmc":
        sobol = rng.random() < 0.5
        return dict(kind=kind, levels=rng.randint(2, 6), base_steps=rng.choice((4, 8, 16)),
                    paths=size(4_000, 200_000), sampling="scrambled_sobol" if sobol else "counter_hash",
                    replicates=4 if sobol else 1)
    if kind == "greeks":
        estimator = rng.choice(("bump_and_revalue", "bump_and_revalue", "pathwise", "likelihood_ratio"))
        if estimator != "bump_and_revalue":
            return dict(kind=kind, workload="european_call", paths=size(4_000, 4_000_000), steps=1,
                        sampling="pseudorandom", technique="standard", estimator=estimator,
                        precision=rng.choice(("fp32_path", "fp64_plain")))
        return dict(kind=kind, paths=size(4_000, 262_144), steps=rng.randint(16, 128),
                    workload=rng.choice(("arithmetic_asian_call", "down_and_out_call", "lookback_call")),
                    sampling=rng.choice(("scrambled_sobol", "counter_hash", "pseudorandom")),
                    technique=rng.choice(techniques), precision="fp32_path", estimator=estimator)
    return dict(kind=kind, paths=size(4_000, 2_000_000), threads=rng.choice((1, 1, 4)))


def configs(case, seed):
    """The (workload, config) pairs of a case: sizes from the case, market data from the seed."""
    rng = random.Random(seed)
    kind = case["kind"]

    def market():
        return dict(s0=100.0, k=rng.uniform(90.0, 110.0), r=0.03, sigma=rng.uniform(0.15, 0.35),
                    t=rng.uniform(0.5, 1.5), seed=rng.randrange(1 << 32))

    if kind == "terminal":
        return [("european_call", dict(market(), n_paths=case["paths"], technique=case["technique"],
                                       sampling=case["sampling"]))]
    if kind == "gbm_fp64":
        return [(case["workload"], dict(market(), method="stepwise", n_paths=case["paths"], n_steps=case["steps"],
                                        n_threads=case["threads"], technique=case["technique"], barrier=80.0,
                                        precision="fp64_plain"))]
    if kind == "exotics":
        size = dict(n_paths=case["paths"], n_steps=case["steps"])
        return [
            ("european_call", dict(market(), method="stepwise", technique="antithetic", **size)),
            ("arithmetic_asian_call", dict(market(), technique="control_variate", **size)),
            ("down_and_out_call", dict(market(), barrier=80.0, **size)),
            ("lookback_call", dict(market(), **size)),
            ("basket_call", dict(market(), method="stepwise", **size, **BASKET5)),
            ("european_call", dict(market(), model="heston", **HESTON, **size)),
        ]
    if kind == "structured":
        size = dict(method="stepwise", n_paths=case["paths"], n_steps=case["steps"], precision=case["precision"])
        return [("european_call", dict(market(), sampling="randomized_halton", **size)),
                ("arithmetic_asian_call", dict(market(), sampling="latin_hypercube", **size)),
                ("lookback_call", dict(market(), sampling="scrambled_sobol_brownian_bridge", **size))]
    if kind == "pair":
        size = dict(n_paths=case["paths"], n_steps=case["steps"], sampling="scrambled_sobol",
                    precision=case["precision"])
        return [("european_call", dict(market(), model="heston", **HESTON, **size)),
                ("european_call", dict(market(), model="merton", method="stepwise", jump_intensity=0.5,
                                       jump_mean=-0.1, jump_volatility=0.15, **size))]
    if kind == "lsm":
        size = dict(n_paths=case["paths"], n_steps=case["steps"], basis_degree=case["degree"],
                    precision=case["precision"])
        out = [("american_put", dict(market(), **size, r=0.06))]
        if case["bermudan"]:
            dates = sorted({max(1, case["steps"] * q // 8) for q in range(1, 9)})
            out.append(("bermudan_put", dict(market(), **size, r=0.06, exercise_steps=dates)))
        return out
    if kind == "book":
        sizes = random.Random(case["sizes"])
        out = []
        for i in range(case["contracts"]):
            workload = BOOK_KINDS[i % 4]
            paths = int(round(math.exp(sizes.uniform(math.log(1e3), math.log(1e6)))))
            k, sigma = rng.uniform(50.0, 150.0), rng.uniform(0.1, 0.6)
            cfg = dict(s0=100.0, k=k, r=0.03, sigma=sigma, t=rng.uniform(0.1, 2.0), seed=rng.randrange(1 << 32),
                       n_paths=paths, n_steps=sizes.randint(16, 365), sampling="counter_hash", method="stepwise")
            if workload == "up_and_out_call":
                cfg["barrier"] = rng.uniform(1.1, 1.5) * max(100.0, k)
            if workload == "basket_call":
                cfg.update(spots=[100.0] * 5, sigmas=[sigma] * 5, weights=[0.2] * 5, corr=0.3)
            out.append((workload, cfg))
        return out
    if kind == "mlmc":
        return [("arithmetic_asian_mlmc", dict(market(), levels=case["levels"], base_steps=case["base_steps"],
                                               refinement_factor=2, scramble_replicates=case["replicates"],
                                               paths_per_level=[max(2, case["paths"] >> i)
                                                                for i in range(case["levels"])],
                                               sampling=case["sampling"]))]
    if kind == "greeks":
        return [(case["workload"], dict(market(), n_paths=case["paths"], n_steps=case["steps"], barrier=80.0,
                                        sampling=case["sampling"], technique=case["technique"],
                                        precision=case["precision"]))]
    return [("european_call", dict(market(), model="merton", n_paths=case["paths"], n_threads=case["threads"],
                                   jump_intensity=0.4, jump_mean=-0.08, jump_volatility=0.25))]


def prepare(case, seed):
    backend = native.backend()
    reqs = [make_request(workload, cfg) for workload, cfg in configs(case, seed)]
    if case["kind"] == "pair" and case["precision"] == "fp32_path":
        for req in reqs:  # a program that prices one shape over and over has its launch shape measured
            backend.prepare(req)
    return dict(backend=backend, reqs=reqs, estimator=case.get("estimator"), lsm=case["kind"] == "lsm")


def run(state):
    backend, reqs = state["backend"], state["reqs"]
    if state["estimator"]:
        rep = backend.greeks(reqs[0], state["estimator"])
        return dict(base_price=rep.base_price, base_stderr=rep.base_stderr,
                    estimates=[dict(value=e.value, stderr=e.stderr, up=e.bumped_up_price, down=e.bumped_down_price)
                               for e in rep.estimates[: rep.n_estimates]])
    results = [backend.price(reqs[0])] if len(reqs) == 1 else backend.price_batch(reqs)
    out = []
    for res in results:
        row = dict(price=res.price, stderr=res.stderr)
        if state["lsm"]:
            row.update(early=res.early_exercise_count, maturity=res.maturity_exercise_count)
        if res.n_levels:
            row["level_mean"] = list(res.level_mean[: res.n_levels])
        out.append(row)
    return out


# A standard normal counts 24 operations and each step its update (the
# benchmark's convention: Heston 16, Merton 4), an exponential 8.
def work(case):
    flops = 0.0
    cfgs = configs(case, 0)
    for workload, cfg in cfgs:
        if workload == "arithmetic_asian_mlmc":
            fine = [cfg["base_steps"] * 2**i for i in range(cfg["levels"])]
            flops += sum(p * f * 48.0 for p, f in zip(cfg["paths_per_level"], fine)) * cfg["scramble_replicates"]
            continue
        units = cfg["n_paths"]
        model = cfg.get("model", "gbm")
        steps = cfg.get("n_steps", 1)
        per = 28.0
        if model == "heston":
            per = 64.0
        elif workload == "basket_call":
            per = 5 * 28.0
        elif workload in ("arithmetic_asian_call", "lookback_call", "american_put", "bermudan_put"):
            per = 36.0
        if workload in ("american_put", "bermudan_put"):
            per += 40.0  # the date's regression
        if case["kind"] == "greeks":
            per = 24.0 + 9 * (per - 24.0) * (2 if cfg["technique"] == "antithetic" else 1)
            units = (units + 1) // 2 if cfg["technique"] == "antithetic" else units
        flops += units * steps * per
    return dict(bytes=2048.0 * len(cfgs), flops=flops)


# ----------------------------------------------- the same estimates in FP64 ---
DEV = "cuda" if torch.cuda.is_available() else "cpu"
M32 = 0xFFFFFFFF
M64 = (1 << 64) - 1
TINY = 2.2250738585072014e-308


def s64(x):
    """A 64-bit word as the int64 torch holds it in."""
    x &= M64
    return x - (1 << 64) if x >> 63 else x


def shr(x, k):
    """Logical right shift of int64 words."""
    return (x >> k) & ((1 << (64 - k)) - 1)


def splitmix(x):
    x = (x + 0x9E3779B97F4A7C15) & M64
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & M64
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & M64
    return x ^ (x >> 31)


def splitmix_t(x):
    x = x + s64(0x9E3779B97F4A7C15)
    x = (x ^ shr(x, 30)) * s64(0xBF58476D1CE4E5B9)
    x = (x ^ shr(x, 27)) * s64(0x94D049BB133111EB)
    return x ^ shr(x, 31)


def open01(x):
    """53-bit uniforms of int64 words, never 0."""
    return torch.clamp(shr(x, 11).double() * 2.0**-53, min=TINY)


def xorshift_step(x):
    x = x ^ (x >> 12)
    x = (x ^ (x << 25)) & M64
    return x ^ (x >> 27)


def columns(run):
    """The images of the 64 basis states under `run` steps."""
    out = []
    for i in range(64):
        x = 1 << i
        for _ in range(run):
            x = xorshift_step(x)
        out.append(x)
    return out


def apply_columns(cols, x):
    y = 0
    for i in range(64):
        if (x >> i) & 1:
            y ^= cols[i]
    return y


def stream(seed, count, run=64):
    """The first `count` outputs of the reference's xorshift64* stream: the
    states 0, run, 2 run, ... by doubling, then `run` steps of all of them."""
    seed = seed or 0x9E3779B97F4A7C15
    runs = -(-count // run)
    state = torch.tensor([s64(seed)], dtype=torch.int64, device=DEV)
    cols = columns(run)  # the jump over the states already there
    while state.numel() < runs:
        host = [[0] * 256 for _ in range(8)]
        for b in range(8):
            for v in range(1, 256):
                low = v & -v
                host[b][v] = host[b][v ^ low] ^ cols[8 * b + low.bit_length() - 1]
        table = torch.tensor([[s64(v) for v in row] for row in host], dtype=torch.int64, device=DEV)
        more = torch.zeros_like(state)
        for b in range(8):
            more ^= table[b][(state >> (8 * b)) & 255]
        state = torch.cat([state, more])
        cols = [apply_columns(cols, c) for c in cols]
    state = state[:runs].clone()
    out = torch.empty(runs, run, dtype=torch.int64, device=DEV)
    for i in range(run):
        state = state ^ shr(state, 12)
        state = state ^ (state << 25)
        state = state ^ shr(state, 27)
        out[:, i] = state * s64(0x2545F4914F6CDD1D)
    return out.view(-1)[:count]


def box_muller(words):
    """Both normals of each pair of stream outputs, in order."""
    u = open01(words).view(-1, 2)
    radius = torch.sqrt(-2.0 * torch.log(u[:, 0]))
    angle = 2.0 * math.pi * u[:, 1]
    return torch.stack([radius * torch.cos(angle), radius * torch.sin(angle)], 1).view(-1)


def brev(x):
    for s, m in ((1, 0x55555555), (2, 0x33333333), (4, 0x0F0F0F0F), (8, 0x00FF00FF)):
        x = ((x >> s) & m) | ((x & m) << s)
    return ((x >> 16) | (x << 16)) & M32


def owen(x, seed):
    """Burley's hash-based nested scramble of 32-bit words; `seed` a tensor or a number."""
    x = (brev(x) + seed) & M32
    for c in (0x6C50B47C, 0xB82F1E52, 0xC7AFE638, 0x8D22F6E6):
        x = x ^ ((x * c) & M32)
    return brev(x)


@lru_cache(maxsize=None)
def directions():
    """Joe-Kuo direction numbers [256][32]: torch's Sobol engine holds the first
    30; each dimension's primitive polynomial, found from them, gives two more."""
    state = torch.quasirandom.SobolEngine(256).sobolstate.numpy().astype(np.int64) << 2
    out = np.zeros((256, 32), dtype=np.int64)
    out[:, :30] = state
    out[0] = 1 << (31 - np.arange(32))
    for d in range(1, 256):
        v = state[d]
        for s in range(1, 14):
            a = np.arange(1 << (s - 1))  # the inner coefficients, highest first

            def term(j):
                t = np.full(a.shape, out[d, j - s] ^ (out[d, j - s] >> s))
                for i in range(1, s):
                    t ^= np.where((a >> (s - 1 - i)) & 1, out[d, j - i], 0)
                return t

            fits = np.ones(a.shape, dtype=bool)
            for j in range(s, 30):
                fits &= term(j) == v[j]
            if fits.sum() == 1:
                which = int(np.argmax(fits))
                for j in (30, 31):
                    out[d, j] = term(j)[which]
                break
        else:
            raise ValueError("no polynomial for Sobol dimension %d" % d)
    return out


@lru_cache(maxsize=None)
def direction_tables():
    v = directions()
    t = np.zeros((256, 4, 256), dtype=np.int64)
    for b in range(4):
        for bit in range(8):
            on = ((np.arange(256) >> bit) & 1).astype(bool)
            t[:, b, on] ^= v[:, 8 * b + bit][:, None]
    return torch.tensor(t, device=DEV)


def primes(count):
    out, c = [], 2
    while len(out) < count:
        if all(c % p for p in out if p * p <= c):
            out.append(c)
        c += 1
    return out


def inverse_normal(p):
    """The reference's rational inverse normal (Acklam), in FP64."""
    a = (-3.969683028665376e1, 2.209460984245205e2, -2.759285104469687e2, 1.38357751867269e2, -3.066479806614716e1,
         2.506628277459239)
    b = (-5.447609879822406e1, 1.615858368580409e2, -1.556989798598866e2, 6.680131188771972e1, -1.328068155288572e1)
    c = (-7.784894002430293e-3, -3.223964580411365e-1, -2.400758277161838, -2.549732539343734, 4.374664141464968,
         2.938163982698783)
    d = (7.784695709041462e-3, 3.224671290700398e-1, 2.445134137142996, 3.754408661907416)

    def poly(cs, x):
        acc = torch.full_like(x, cs[0])
        for k in cs[1:]:
            acc = acc * x + k
        return acc

    p = torch.clamp(p, TINY, 1.0 - 2.0**-52)
    q = p - 0.5
    r = q * q
    mid = poly(a, r) * q / poly(b + (1.0,), r)
    t = torch.sqrt(-2.0 * torch.log(torch.where(p < 0.5, p, 1.0 - p)))
    tail = poly(c, t) / poly(d + (1.0,), t)
    return torch.where(p < 0.02425, tail, torch.where(p > 1.0 - 0.02425, -tail, mid))


class Samples:
    """Normals (and raw uniforms) of every point by dimension: normal(d), uniform(d)."""

    def __init__(self, sampling, seed, points, dims, threads=1, paths=None):
        self.kind, self.seed, self.n, self.dims = sampling, seed, points, dims
        self.point = torch.arange(points, device=DEV)
        if sampling == "pseudorandom":
            chunks = threads if threads > 1 and points >= 2000 * threads else 1
            base, rem = divmod(points, chunks)
            z = []
            for c in range(chunks):
                need = (base + (c < rem)) * dims
                chunk_seed = splitmix((seed + c * 0x9E3779B97F4A7C15) & M64) if chunks > 1 else seed
                z.append(box_muller(stream(chunk_seed, 2 * (-(-need // 2))))[:need])
            self.z = torch.cat(z).view(points, dims)
        elif sampling == "randomized_halton":
            self.primes = primes(max(dims, 2))
        elif sampling == "latin_hypercube":
            self.paths = paths or points

    def sobol(self, d):
        block = self.point >> 16
        dim, group = d & 255, d >> 8
        seed = ((self.seed & M32) + group + block * 0x9E3779B9) & M32
        index = owen(self.point & 0xFFFF, seed)
        table = direction_tables()[dim]
        x = table[0][index & 255] ^ table[1][(index >> 8) & 255] ^ table[2][(index >> 16) & 255] ^ table[3][index >> 24]
        out_seed = seed ^ ((dim + 0x9E3779B9 + (seed << 6) + (seed >> 2)) & M32)
        return owen(x, out_seed)

    def counter(self, d, lane):
        x = (self.point * 747796405) & M32
        x = x ^ ((self.seed & M32) ^ ((d * 2891336453) & M32) ^ ((lane * 277803737) & M32))
        x = (x + 0x9E3779B9) & M32
        x = ((x ^ (x >> 16)) * 0x85EBCA6B) & M32
        x = ((x ^ (x >> 13)) * 0xC2B2AE35) & M32
        x = x ^ (x >> 16)
        return ((x + 1).double() / 4294967297.0).float().double()

    def halton(self, d):
        base = self.primes[d]
        index, f, value = self.point + 1, 1.0 / base, torch.zeros(self.n, dtype=torch.float64, device=DEV)
        top = self.n
        while top > 0:
            value += f * (index % base).double()
            index = index // base
            top //= base
            f /= base
        shift = max((splitmix((self.seed + d * 0x9E3779B97F4A7C15) & M64) >> 11) * 2.0**-53, TINY)
        shifted = torch.clamp(value, min=TINY) + shift
        return shifted - torch.floor(shifted)

    def latin(self, d):
        n = self.paths
        mixed = splitmix(self.seed ^ ((d * 0x9E3779B97F4A7C15) & M64) ^ 0xD1B54A32D192ED03)
        c = 1
        if n > 1:
            c = max(mixed % n, 1)
            c += 1 - c % 2
            while math.gcd(c, n) != 1:
                c += 2
                if c >= n:
                    c = 1
        offset = splitmix(mixed ^ 0xA24BAED4963EE407) % n
        jitter_seed = s64(splitmix(mixed ^ 0x9FB21C651E98DF25))
        stratum = (c * self.point + offset) % n
        jitter = open01(splitmix_t(jitter_seed ^ (self.point * s64(0xBF58476D1CE4E5B9))))
        return torch.clamp((stratum.double() + jitter) / n, TINY, 1.0 - 2.0**-52)

    def uniform(self, d):
        if self.kind.startswith("scrambled_sobol"):
            return ((self.sobol(d) >> 9).double() + 0.5) * 2.0**-23
        if self.kind == "counter_hash":
            return self.counter(d, 0)
        return self.halton(d) if self.kind == "randomized_halton" else self.latin(d)

    def normal(self, d):
        if self.kind == "pseudorandom":
            return self.z[:, d]
        if self.kind == "counter_hash":
            return torch.sqrt(-2.0 * torch.log(self.counter(d, 0))) * torch.cos(2.0 * math.pi * self.counter(d, 1))
        return inverse_normal(self.uniform(d))


def bridge(samples, steps, maturity):
    """The step normals of a Brownian-bridge path, as a list by step."""
    dt = maturity / steps
    w = {0: torch.zeros(samples.n, dtype=torch.float64, device=DEV), steps: math.sqrt(maturity) * samples.normal(0)}
    todo, dim = [(0, steps)], 1
    while todo:
        left, right = todo.pop()
        if right <= left + 1:
            continue
        mid = (left + right) // 2
        tl, tm, tr = left * dt, mid * dt, right * dt
        w[mid] = ((tr - tm) / (tr - tl) * w[left] + (tm - tl) / (tr - tl) * w[right]
                  + math.sqrt((tm - tl) * (tr - tm) / (tr - tl)) * samples.normal(dim))
        dim += 1
        todo += [(mid, right), (left, mid)]
    return [(w[i + 1] - w[i]) / math.sqrt(dt) for i in range(steps)]


def poisson(u, mean):
    """Jump counts by inversion of the uniforms."""
    prob = total = math.exp(-mean)
    count = torch.zeros(u.numel(), dtype=torch.float64, device=DEV)
    for k in range(1, 60):
        more = u > total
        if not bool(more.any()):
            break
        count += more
        prob *= mean / k
        total += prob
    return count


def units_of(cfg):
    return (cfg["n_paths"] + 1) // 2 if cfg.get("technique") == "antithetic" else cfg["n_paths"]


def sample_set(workload, cfg):
    """The samples of a request; a bump leg uses the base request's."""
    model, steps = cfg.get("model", "gbm"), cfg.get("n_steps", 1)
    stepwise = cfg.get("method") == "stepwise" or workload != "european_call" or model == "heston"
    steps = steps if stepwise else 1
    per = {"heston": 2, "merton": 3}.get(model, len(cfg["spots"]) if workload == "basket_call" else 1)
    threads = cfg.get("n_threads", 1)
    if workload == "european_call" and cfg.get("technique") == "antithetic" or workload == "basket_call":
        threads = 1  # the reference runs these on one stream
    return Samples(cfg.get("sampling", "pseudorandom"), cfg["seed"], units_of(cfg), steps * per, threads,
                   cfg["n_paths"])


def path_payoffs(workload, cfg, smp):
    """Discounted payoffs and discounted control of every unit."""
    model, technique = cfg.get("model", "gbm"), cfg.get("technique", "standard")
    k, r, t, sigma = cfg["k"], cfg["r"], cfg["t"], cfg["sigma"]
    disc = math.exp(-r * t)
    zero = torch.zeros(smp.n, dtype=torch.float64, device=DEV)
    if workload == "basket_call":
        return basket_payoffs(cfg, smp)
    ls0 = math.log(cfg["s0"])
    if model == "merton":
        return merton_step_payoffs(cfg, smp)
    sides = (1.0, -1.0) if technique == "antithetic" else (1.0,)
    stepwise = cfg.get("method") == "stepwise" or workload != "european_call" or model == "heston"
    steps = cfg["n_steps"] if stepwise else 1
    dt = t / steps
    ls = [zero + ls0 for _ in sides]
    v = [zero + cfg.get("v0", 0.0) for _ in sides]
    acc = [zero + (cfg["s0"] if workload == "lookback_call" else 0.0) for _ in sides]
    barrier = cfg.get("barrier", 0.0)
    out = [zero.bool() | (workload == "down_and_out_call" and cfg["s0"] <= barrier)
           | (workload == "up_and_out_call" and cfg["s0"] >= barrier) for _ in sides]
    z_of = smp.normal
    if smp.kind == "scrambled_sobol_brownian_bridge":
        z_of = bridge(smp, steps, t).__getitem__
    for s in range(steps):
        z = z_of(2 * s if model == "heston" else s)
        zi = smp.normal(2 * s + 1) if model == "heston" else None
        for i, sign in enumerate(sides):
            if model == "heston":
                root = torch.sqrt(v[i])
                zp = cfg["rho"] * z + math.sqrt(max(1.0 - cfg["rho"] ** 2, 0.0)) * zi
                ls[i] = ls[i] + (r - 0.5 * v[i]) * dt + root * math.sqrt(dt) * (sign * zp)
                v[i] = torch.clamp(v[i] + cfg["kappa"] * (cfg["theta"] - v[i]) * dt
                                   + cfg["vol_of_vol"] * root * math.sqrt(dt) * (sign * z), min=0.0)
            else:
                ls[i] = ls[i] + ((r - 0.5 * sigma * sigma) * dt + sigma * math.sqrt(dt) * (sign * z))
            if workload == "arithmetic_asian_call":
                acc[i] = acc[i] + torch.exp(ls[i])
            elif workload == "lookback_call":
                acc[i] = torch.maximum(acc[i], torch.exp(ls[i]))
            elif workload == "down_and_out_call":
                out[i] = out[i] | (torch.exp(ls[i]) <= barrier)
            elif workload == "up_and_out_call":
                out[i] = out[i] | (torch.exp(ls[i]) >= barrier)
    pay = []
    for i in range(len(sides)):
        level = {"arithmetic_asian_call": acc[i] / steps, "lookback_call": acc[i]}.get(workload, torch.exp(ls[i]))
        pay.append(torch.where(out[i], zero, torch.clamp(level - k, min=0.0)) * disc)
    return sum(pay) / len(pay), disc * torch.exp(ls[0])


def basket_payoffs(cfg, smp):
    d, steps = len(cfg["spots"]), cfg["n_steps"]
    dt = cfg["t"] / steps
    corr = np.full((d, d), cfg["corr"])
    np.fill_diagonal(corr, 1.0)
    chol = np.linalg.cholesky(corr)
    x = [torch.zeros(smp.n, dtype=torch.float64, device=DEV) for _ in range(d)]
    for s in range(steps):
        z = [smp.normal(s * d + a) for a in range(d)]
        for a in range(d):
            zc = sum(float(chol[a, b]) * z[b] for b in range(a + 1))
            sg = cfg["sigmas"][a]
            x[a] = x[a] + ((cfg["r"] - 0.5 * sg * sg) * dt + sg * math.sqrt(dt) * zc)
    weights = cfg.get("weights", [1.0 / d] * d)
    basket = sum(weights[a] * (cfg["spots"][a] * torch.exp(x[a])) for a in range(d))
    disc = math.exp(-cfg["r"] * cfg["t"])
    return torch.clamp(basket - cfg["k"], min=0.0) * disc, basket * disc


def merton_step_payoffs(cfg, smp):
    steps = cfg["n_steps"]
    dt, jm, jv = cfg["t"] / steps, cfg["jump_mean"], cfg["jump_volatility"]
    kj = cfg["jump_intensity"] * (math.exp(jm + 0.5 * jv * jv) - 1.0)
    drift, vol = (cfg["r"] - kj - 0.5 * cfg["sigma"] ** 2) * dt, cfg["sigma"] * math.sqrt(dt)
    ls = torch.full((smp.n,), math.log(cfg["s0"]), dtype=torch.float64, device=DEV)
    for s in range(steps):
        n = poisson(smp.uniform(3 * s + 1), cfg["jump_intensity"] * dt)
        ls = ls + (drift + vol * smp.normal(3 * s)) + (n * jm + jv * torch.sqrt(n) * smp.normal(3 * s + 2))
    disc = math.exp(-cfg["r"] * cfg["t"])
    st = torch.exp(ls)
    return torch.clamp(st - cfg["k"], min=0.0) * disc, st * disc


def merton_replay_payoffs(cfg):
    """The terminal Merton paths of the reference's sequential streams: a path
    draws a normal (one may be cached), a uniform, and a normal if it jumps."""
    n, threads = cfg["n_paths"], cfg.get("n_threads", 1)
    mean, jm, jv, t = cfg["jump_intensity"] * cfg["t"], cfg["jump_mean"], cfg["jump_volatility"], cfg["t"]
    p0 = math.exp(-mean)
    chunks = threads if threads > 1 and n >= 2000 * threads else 1
    base, rem = divmod(n, chunks)
    pay, ctl = [], []
    for c in range(chunks):
        paths = base + (c < rem)
        seed = splitmix((cfg["seed"] + c * 0x9E3779B97F4A7C15) & M64) if chunks > 1 else cfg["seed"]
        u = open01(stream(seed, 3 * paths + 8))
        jump = (u > p0).cpu().numpy().tobytes()
        pair, which, pois, pair2 = [0] * paths, [0] * paths, [0] * paths, [0] * paths
        at, cached = 0, -1  # cached: where the pair of the cached sine normal was drawn
        for i in range(paths):
            if cached < 0:
                pair[i] = at
                j = at + 2
                pair2[i] = ~at  # the second normal, if any, is this pair's sine
                cached = at
                at += 3
                if jump[j]:
                    cached = -1
            else:
                pair[i], which[i] = cached, 1
                j = at
                cached = -1
                at += 1
                if jump[j]:
                    pair2[i] = at
                    cached = at
                    at += 2
            pois[i] = j
        pair, which, pois, pair2 = (torch.tensor(v, device=DEV) for v in (pair, which, pois, pair2))

        def normal(first, sine):
            radius = torch.sqrt(-2.0 * torch.log(u[first]))
            angle = 2.0 * math.pi * u[first + 1]
            return radius * torch.where(sine, torch.sin(angle), torch.cos(angle))

        z = normal(pair, which.bool())
        count = poisson(u[pois], mean)
        zj = normal(torch.where(pair2 < 0, ~pair2, pair2), pair2 < 0)
        kj = cfg["jump_intensity"] * (math.exp(jm + 0.5 * jv * jv) - 1.0)
        jumps = torch.where(count > 0, count * jm + jv * torch.sqrt(count) * zj, torch.zeros_like(z))
        st = torch.exp(math.log(cfg["s0"]) + (cfg["r"] - kj - 0.5 * cfg["sigma"] ** 2) * t
                       + cfg["sigma"] * math.sqrt(t) * z + jumps)
        disc = math.exp(-cfg["r"] * t)
        pay.append(torch.clamp(st - cfg["k"], min=0.0) * disc)
        ctl.append(st * disc)
    return torch.cat(pay), torch.cat(ctl)


def estimate(workload, cfg, pay, ctl):
    """(price, standard error) of the payoffs under the request's technique."""
    n = pay.numel()
    mean, square = float(pay.mean()), float((pay * pay).mean())
    if cfg.get("technique") == "control_variate":
        c, cc, pc = float(ctl.mean()), float((ctl * ctl).mean()), float((pay * ctl).mean())
        beta = (pc - mean * c) / (cc - c * c)
        e = cfg["s0"]
        adjusted = pay - beta * (ctl - e)
        mean, square = float(adjusted.mean()), float((adjusted * adjusted).mean())
    return mean, math.sqrt(max(square - mean * mean, 0.0)) / math.sqrt(n)


def lsm_exact(workload, cfg):
    n, steps, k = cfg["n_paths"], cfg["n_steps"], cfg["k"]
    dt = cfg["t"] / steps
    smp = Samples("pseudorandom", cfg["seed"], n, steps)
    s, path = torch.full((n,), cfg["s0"], dtype=torch.float64, device=DEV), []
    for i in range(steps):
        s = s * torch.exp((cfg["r"] - 0.5 * cfg["sigma"] ** 2) * dt + cfg["sigma"] * math.sqrt(dt) * smp.normal(i))
        path.append(s)
    dates = cfg.get("exercise_steps") or list(range(1, steps + 1))
    cash = torch.clamp(k - path[-1], min=0.0)
    when = torch.full((n,), steps, dtype=torch.int64, device=DEV)
    disc = torch.exp(torch.arange(steps + 1, dtype=torch.float64, device=DEV) * (-cfg["r"] * dt))
    for date in reversed([d for d in dates if d < steps]):
        s = path[date - 1]
        x = s / k
        basis = torch.stack([torch.ones_like(x), 1 - x, 1 - 2 * x + 0.5 * x * x,
                             1 - 3 * x + 1.5 * x * x - x**3 / 6][: cfg["basis_degree"] + 1], 1)
        money = k - s > 0
        a = basis[money]
        if a.shape[0] < a.shape[1]:
            continue
        b = (cash * disc[when - date])[money]
        beta = torch.linalg.solve(a.T @ a, a.T @ b)
        early = money & (k - s > torch.clamp(basis @ beta, min=0.0))
        cash = torch.where(early, k - s, cash)
        when = torch.where(early, torch.full_like(when, date), when)
    value = cash * disc[when]
    mean = float(value.mean())
    se = math.sqrt(max(float((value * value).mean()) - mean * mean, 0.0)) / math.sqrt(n)
    if workload == "american_put" and max(k - cfg["s0"], 0.0) > mean:
        mean, se = max(k - cfg["s0"], 0.0), 0.0
    return dict(price=mean, stderr=se, early=None, maturity=None)


def mlmc_exact(cfg):
    k, r, t, sigma, levels = cfg["k"], cfg["r"], cfg["t"], cfg["sigma"], cfg["levels"]
    pseudo = cfg["sampling"] in ("pseudorandom", "counter_hash")
    reps = 1 if pseudo else cfg["scramble_replicates"]
    disc, prices, means, se = math.exp(-r * t), [], [[] for _ in range(levels)], 0.0
    for rep in range(reps):
        seed = splitmix((cfg["seed"] + rep * 0x9E3779B97F4A7C15) & M64) if reps > 1 else cfg["seed"]
        price, var = 0.0, 0.0
        for level in range(levels):
            fine, paths = cfg["base_steps"] * 2**level, cfg["paths_per_level"][level]
            smp = Samples(cfg["sampling"], splitmix((seed + level * 0x9E3779B97F4A7C15) & M64), paths, fine)
            zero = torch.zeros(paths, dtype=torch.float64, device=DEV)
            fl, cl, fs, cs, zsum = zero + math.log(cfg["s0"]), zero + math.log(cfg["s0"]), zero, zero, zero
            fdt, cdt = t / fine, 2 * t / fine
            for s in range(fine):
                z = smp.normal(s)
                fl = fl + ((r - 0.5 * sigma**2) * fdt + sigma * math.sqrt(fdt) * z)
                fs = fs + torch.exp(fl)
                zsum = zsum + z
                if level and s % 2:
                    cl = cl + ((r - 0.5 * sigma**2) * cdt + sigma * math.sqrt(cdt) * zsum / math.sqrt(2.0))
                    cs, zsum = cs + torch.exp(cl), zero
            pay = torch.clamp(fs / fine - k, min=0.0) * disc
            if level:
                pay = pay - torch.clamp(cs / (fine // 2) - k, min=0.0) * disc
            mean = float(pay.mean())
            means[level].append(mean)
            price += mean
            var += max(float((pay * pay).mean()) - mean * mean, 0.0) / paths
        prices.append(price)
        se = math.sqrt(var)
    price = sum(prices) / reps
    if reps > 1:
        se = math.sqrt(sum((p - price) ** 2 for p in prices) / (reps - 1) / reps)
    return dict(price=price, stderr=se, level_mean=[sum(m) / reps for m in means])


def greeks_exact(case, workload, cfg):
    smp = sample_set(workload, cfg)
    if case["estimator"] == "bump_and_revalue":
        price, se = estimate(workload, cfg, *path_payoffs(workload, cfg, smp))
        out = []
        for field, bump, sign in (("s0", max(cfg["s0"] * 0.01, 0.01), 1), ("sigma", max(cfg["sigma"] * 0.05, 0.005), 1),
                                  ("r", 0.001, 1), ("t", min(1.0 / 365.0, 0.25 * cfg["t"]), -1)):
            up, up_se = estimate(workload, *leg(workload, cfg, smp, field, cfg[field] + bump))
            down, down_se = estimate(workload, *leg(workload, cfg, smp, field, cfg[field] - bump))
            out.append(dict(value=sign * (up - down) / (2.0 * bump), stderr=math.hypot(up_se, down_se) / (2.0 * bump),
                            up=up, down=down))
        return dict(base_price=price, base_stderr=se, estimates=out)
    price, se = estimate(workload, cfg, *path_payoffs(workload, cfg, smp))
    s0, k, r, t, sigma = (cfg[f] for f in ("s0", "k", "r", "t", "sigma"))
    z, root, disc = smp.normal(0), math.sqrt(t), math.exp(-r * t)
    s = s0 * torch.exp((r - 0.5 * sigma**2) * t + sigma * root * z)
    pay, live = torch.clamp(s - k, min=0.0), s > k
    if case["estimator"] == "pathwise":
        zero = torch.zeros_like(s)
        slope = s * (r - 0.5 * sigma**2 + sigma * z / (2.0 * root))
        g = [torch.where(live, disc * s / s0, zero), torch.where(live, disc * s * (root * z - sigma * t), zero),
             torch.where(live, disc * (t * s - t * pay), -t * disc * pay),
             -torch.where(live, disc * (slope - r * pay), -r * disc * pay)]
    else:
        g = [disc * pay * z / (s0 * sigma * root), disc * pay * ((z * z - 1.0) / sigma - root * z),
             disc * pay * (z / (sigma * root) - t)]
    return dict(base_price=price, base_stderr=se,
                estimates=[dict(value=float(v.mean()), stderr=math.sqrt(float(v.var()) / v.numel()), up=None, down=None)
                           for v in g])


def leg(workload, cfg, smp, field, value):
    moved = dict(cfg, **{field: value})
    return (moved, *path_payoffs(workload, moved, smp))


def exact(case, seed):
    out = []
    for workload, cfg in configs(case, seed):
        if case["kind"] == "lsm":
            out.append(lsm_exact(workload, cfg))
        elif case["kind"] == "mlmc":
            out.append(mlmc_exact(cfg))
        elif case["kind"] == "greeks":
            return greeks_exact(case, workload, cfg)
        else:
            if case["kind"] == "merton":
                pay, ctl = merton_replay_payoffs(cfg)
            else:
                pay, ctl = path_payoffs(workload, cfg, sample_set(workload, cfg))
            price, se = estimate(workload, cfg, pay, ctl)
            out.append(dict(price=price, stderr=se))
    return out
