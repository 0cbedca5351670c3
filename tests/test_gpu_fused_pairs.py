"""Fused FP32 units that draw their normals two at a time, per path against
the FP64 oracle on the same samples: odd and even steps (a last single
normal), odd stream positions, every asset count of a basket, chunk edges
inside a warp.  FP32 paths: the tolerance of the other FP32 per-path tests
(steps of a log price of 4.6, last place 4.8e-7, at S of 100 to 200)."""

import numpy as np
import pytest

from montepath_b200.requests import make_request
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [
    ("european_call", dict(method="stepwise")),
    ("european_call", dict(model="heston", kappa=2.0, vol_of_vol=0.5, rho=-0.7)),
    ("arithmetic_asian_call", dict(technique="antithetic")),
    ("lookback_call", dict(technique="control_variate")),
]


def check(backend, workload, kw):
    _, ref = O.price_paths(make_request(workload, dict(kw, precision="fp64_plain")))
    got = backend.price_paths(make_request(workload, dict(kw, precision="fp32_path")))
    assert np.allclose(got, ref, rtol=1e-3, atol=2e-3), float(np.max(np.abs(got - ref)))


@pytest.mark.parametrize("workload,kw", CASES)
@pytest.mark.parametrize("sampling", ["pseudorandom", "counter_hash"])
@pytest.mark.parametrize("n_paths,n_steps,threads", [(1, 1, 1), (33, 2, 1), (515, 3, 1), (8003, 36, 4)])
def test_units_by_pairs(backend, workload, kw, sampling, n_paths, n_steps, threads):
    check(backend, workload, dict(kw, sampling=sampling, n_paths=n_paths, n_steps=n_steps, n_threads=threads, seed=13))


@pytest.mark.parametrize("workload", ["european_call", "arithmetic_asian_call", "lookback_call"])
@pytest.mark.parametrize("sampling", ["randomized_halton", "latin_hypercube"])
@pytest.mark.parametrize("n_paths,n_steps", [(1, 1), (8, 2), (243, 5), (8003, 36)])
def test_lattice_units_by_pairs(backend, workload, sampling, n_paths, n_steps):
    """Pairs of dimensions (of different digit counts, and a last single one)
    against paths of the same FP32 normals, which the sampler gives one at a
    time: only the path's own FP32 rounding is between them."""
    req = make_request(workload, dict(method="stepwise", sampling=sampling, n_paths=n_paths, n_steps=n_steps, seed=13,
                                      precision="fp32_path"))
    z = backend.generate_normals(req.sampling, 13, n_paths, n_steps, fp32=True).astype(np.float64)
    z = z.reshape(n_paths, n_steps)
    dt = req.t / n_steps
    log = np.log(req.s0) + np.cumsum((req.r - 0.5 * req.sigma**2) * dt + req.sigma * np.sqrt(dt) * z, axis=1)
    spot = np.exp(log)
    level = {"european_call": spot[:, -1], "arithmetic_asian_call": spot.mean(axis=1),
             "lookback_call": np.maximum(spot.max(axis=1), req.s0)}[workload]
    ref = np.exp(-req.r * req.t) * np.maximum(level - req.k, 0.0)
    got = backend.price_paths(req)
    assert np.allclose(got, ref, rtol=1e-3, atol=2e-3), float(np.max(np.abs(got - ref)))


@pytest.mark.parametrize("assets", range(1, 9))
@pytest.mark.parametrize("n_steps", [1, 2, 5])
@pytest.mark.parametrize("sampling,technique", [("pseudorandom", "standard"), ("counter_hash", "antithetic")])
def test_baskets_by_pairs(backend, assets, n_steps, sampling, technique):
    corr = [[1.0 if i == j else 0.25 for j in range(assets)] for i in range(assets)]
    check(backend, "basket_call", dict(method="stepwise", n_steps=n_steps, n_paths=2001, seed=6, sampling=sampling,
                                       technique=technique, spots=[90.0 + 4.0 * i for i in range(assets)],
                                       sigmas=[0.15 + 0.03 * i for i in range(assets)], corr=corr))


@pytest.mark.parametrize("members", [1, 4, 5])
def test_inline_and_listed_groups(backend, members):
    """Groups of up to four requests travel as launch parameters, larger ones
    through a tile list: the same prices either way, alternating, with more
    tiles than resident blocks and with a single one."""

    reqs = [make_request("european_call", dict(method="stepwise", n_steps=3 + i, seed=i, sampling="counter_hash",
                                               n_paths=(400_001 if i % 2 else 77)))
            for i in range(members)]
    reqs.append(make_request("basket_call", dict(n_paths=5000, seed=1)))
    alone = [backend.price(r) for r in reqs]
    for _ in range(3):
        for a, b in zip(alone, backend.price_batch(reqs)):
            assert (a.price, a.stderr, a.n_samples) == (b.price, b.stderr, b.n_samples)
        for r, a in zip(reqs, alone):
            assert backend.price(r).price == a.price
