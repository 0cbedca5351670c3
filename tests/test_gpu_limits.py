"""Calls at the ends of the ranges the entry points accept."""

import pytest

from montepath_b200.requests import make_request

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sampling", ["counter_hash", "scrambled_sobol", "randomized_halton"])
@pytest.mark.parametrize("workload,kw", [
    ("european_call", dict(method="stepwise")),
    ("european_call", dict(model="heston")),
    ("european_call", dict(model="merton", method="stepwise", jump_intensity=0.5)),
    ("arithmetic_asian_call", {}),
    ("lookback_call", {}),
])
def test_prices_below_the_fp32_normal_range(backend, workload, kw, sampling):
    """A spot of 1e-39 is an FP32 denormal: paths and payoffs keep their
    denormal values.  FP32 against FP64 paths of the same normals.

    Tolerance: the log price is -89.8, where an FP32 addition is off by at most
    3.8e-6 and the scaled exponent by 7.8e-6; 16 steps give 6.1e-5 + 0.8e-5.
    A denormal near 1e-39 is spaced 1.4e-6 of itself; spot, payoff and
    discounted payoff round once each and a strike of a tenth of the spot adds
    a factor of 10 / 9: below 1e-4 in all.
    """
    cfg = dict(kw, s0=1e-39, k=1e-40, n_paths=3001, n_steps=16, seed=11, sampling=sampling)
    want = backend.price(make_request(workload, dict(cfg, precision="fp64_plain"))).price
    got = backend.price(make_request(workload, cfg)).price
    assert abs(got - want) <= 1e-4 * want, (got, want)


MILLION = 1_000_000


@pytest.mark.parametrize("workload,kw,refused,accepted", [
    # samples and half the payoffs; samples and payoffs
    ("european_call", dict(method="stepwise"), 8 * 16 + 4, 8 * 16 + 8),
    # samples, payoffs and half the control values; all of them
    ("european_call", dict(method="stepwise", technique="control_variate"), 8 * 16 + 12, 8 * 16 + 16),
    # three stream positions, their bits and maps, path starts and half the payoffs; all of them
    ("european_call", dict(model="merton", method="terminal"), 26 + 8 + 4, 26 + 8 + 8),
])
def test_budget_counts_every_documented_buffer(workload, kw, refused, accepted):
    """FP64 admission by the documented sizes (bytes per path): the kernels keep
    less in device memory, but the budget a request needs has not changed."""

    from montepath_b200 import abi
    from montepath_b200.backend import BackendError, CudaBackend

    r = make_request(workload, dict(kw, n_paths=MILLION, n_steps=16, sampling="pseudorandom", precision="fp64_plain"))
    with CudaBackend(0, hbm_budget_bytes=refused * MILLION) as small:
        with pytest.raises(BackendError) as err:
            small.price(r)
        assert err.value.status == abi.E_OOM_BUDGET
    with CudaBackend(0, hbm_budget_bytes=accepted * MILLION + (2 << 20)) as enough:  # and the context's own tables
        assert enough.price(r).price > 0.0
        assert enough.price(r).price > 0.0  # beside the buffers of the first call
