"""The one-launch FP64 plain path against the oracle, per path, where its
tiling can go wrong: the last block of a launch, the staged Sobol columns of
few dimensions, several units per thread, and paths shared by several lanes
(odd stream positions, chunk edges inside a warp, every share length).

Tolerance: the device's log, exp and sincospi are within a few units in the
last place of glibc's, a path sums at most 513 of them, and payoffs are of
order 10 to 1000: 1e-11 relative leaves a factor of a hundred.
"""

import numpy as np
import pytest

from montepath_b200 import abi
from montepath_b200.requests import make_request
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def check(backend, workload, **kw):
    r = make_request(workload, dict(kw, precision="fp64_plain"))
    _, ref = O.price_paths(r)
    got = backend.price_paths(r)
    assert np.allclose(got, ref, rtol=1e-11, atol=1e-11), float(np.max(np.abs(got - ref)))
    a, b = backend.price(r), O.price(r)
    assert abs(a.price - b.price) <= 1e-11 * abs(b.price)
    assert abs(a.stderr - b.stderr) <= 1e-9 * abs(b.stderr) + 1e-15
    assert a.n_samples == b.n_samples


@pytest.mark.parametrize("n_steps", [1, 4, 5, 8, 9, 17, 32, 33, 64, 65, 129, 257])
@pytest.mark.parametrize("n_paths", [33, 4097])
def test_plain_sobol_staged_columns(backend, n_steps, n_paths):
    check(backend, "arithmetic_asian_call", n_paths=n_paths, n_steps=n_steps, seed=3, sampling="scrambled_sobol")


@pytest.mark.parametrize("model,n_steps", [("heston", 3), ("heston", 35), ("merton", 3), ("merton", 23), ("merton", 86)])
def test_plain_sobol_quads(backend, model, n_steps):
    check(backend, "european_call", model=model, method="stepwise", n_paths=5001, n_steps=n_steps, seed=9,
          sampling="scrambled_sobol", jump_intensity=3.0)


@pytest.mark.parametrize("kw", [
    dict(sampling="scrambled_sobol"),
    dict(sampling="pseudorandom", technique="control_variate", n_threads=4),
    dict(sampling="latin_hypercube", technique="antithetic"),
])
def test_plain_several_units_per_thread(backend, kw):
    check(backend, "european_call", n_paths=2_200_001, seed=5, **kw)


@pytest.mark.parametrize("workload,technique", [
    ("european_call", "antithetic"),
    ("arithmetic_asian_call", "control_variate"),
    ("down_and_out_call", "antithetic"),
    ("up_and_out_call", "standard"),
    ("lookback_call", "antithetic"),
])
@pytest.mark.parametrize("n_paths,n_steps,threads", [(1, 16, 1), (37, 17, 1), (2501, 63, 1), (2501, 511, 1),
                                                     (8007, 64, 4), (70_001, 33, 8)])
def test_plain_paths_shared_by_lanes(backend, workload, technique, n_paths, n_steps, threads):
    check(backend, workload, method="stepwise", technique=technique, n_paths=n_paths, n_steps=n_steps, seed=21,
          n_threads=threads, barrier=80.0 if workload == "down_and_out_call" else 130.0)


@pytest.mark.parametrize("intensity", [0.0, 1e-9, 900.0])
@pytest.mark.parametrize("precision", ["fp32_path", "fp64_plain"])
def test_sobol_merton_extreme_intensities(backend, intensity, precision):
    """No jump at all, jumps below the 23-bit uniforms' resolution, and exp(-lambda dt) near 0."""

    r = make_request("european_call", dict(model="merton", method="stepwise", n_paths=3000, n_steps=32, seed=4,
                                           jump_intensity=intensity, jump_mean=-0.001, jump_volatility=0.002,
                                           sampling="scrambled_sobol", precision=precision))
    _, ref = O.price_paths(r)
    got = backend.price_paths(r)
    rtol = 1e-11 if precision == "fp64_plain" else 1e-3
    assert np.allclose(got, ref, rtol=rtol, atol=rtol), float(np.max(np.abs(got - ref)))


@pytest.mark.parametrize("sampling", ["randomized_halton", "latin_hypercube"])
@pytest.mark.parametrize("n_paths,n_steps", [(1, 1), (2, 3), (8, 5), (9, 2), (243, 40), (65_536, 3), (65_537, 9)])
def test_lattice_samples_at_digit_edges(backend, sampling, n_paths, n_steps):
    """Point counts at powers of the small primes: the digit count of a
    dimension changes there, and the strata are few.  FP64 normals to the bound
    of the other sampler tests; FP32 ones within normcdfinvf's 5 ulp plus the
    uniform's rounding (the slope of the inverse at 2^-24 is under 2^22)."""

    code = abi.SAMPLINGS[sampling]
    ref = O.generate_normals(code, 7, n_paths, n_steps)
    got = backend.generate_normals(code, 7, n_paths, n_steps)
    assert np.max(np.abs(got - ref) / np.maximum(1.0, np.abs(ref))) < 1e-13
    f32 = backend.generate_normals(code, 7, n_paths, n_steps, fp32=True)
    slope = 1.0 / np.maximum(np.exp(-0.5 * ref * ref) / np.sqrt(2.0 * np.pi), 1e-7)
    assert np.all(np.abs(f32 - ref) < 2e-6 * np.maximum(1.0, np.abs(ref)) + 6e-8 * slope)


def test_halton_wide_digit_products(backend):
    """base^digits past 2^32 (2,700,000 points, primes above 1,626): FP32 against FP64 prices."""

    kw = dict(method="stepwise", n_paths=2_700_000, n_steps=260, seed=3, sampling="randomized_halton")
    a = backend.price(make_request("european_call", dict(kw, precision="fp32_path")))
    b = backend.price(make_request("european_call", dict(kw, precision="fp64_plain")))
    assert abs(a.price - b.price) < 0.01 * b.stderr, (a.price, b.price, b.stderr)


@pytest.mark.parametrize("assets", [1, 2, 5, 8])
@pytest.mark.parametrize("sampling", ["randomized_halton", "latin_hypercube"])
def test_plain_lattice_baskets(backend, assets, sampling):
    """A step's normals drawn in a loop (one asset: without it)."""

    check(backend, "basket_call", method="stepwise", spots=[100.0] * assets, sigmas=[0.2] * assets,
          weights=[1.0 / assets] * assets, corr=0.3, n_paths=1003, n_steps=7, seed=5, sampling=sampling)
