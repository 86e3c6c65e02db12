"""GPU: the path loop's step code at the sizes where it can go wrong, against the oracle on
the same Philox draws.

Tolerances.  FP64: a step on the logarithm of the spot rounds a handful of times at a few
units in the last place (2^-52) of terms below 0.1, so 101 steps stay within 1e-13 of the
oracle; 1e-12 is asserted, as for the other FP64 path checks.  Next to zero variance QE's
(b + Z)^2 loses relative accuracy where b + Z cancels (b >= 0.7, so at most about 1e-12 of
a variance that small moves the spot by far less); 1e-10 on the spot there.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_steps", [1, 2, 15, 16, 17, 101])
@pytest.mark.parametrize("model,scheme", [(m, s) for m in (0, 1) for s in (0, 1, 2)])
def test_fp64_paths_at_block_edges_match_oracle(qk, handle, oracle, model, scheme, n_steps):
    """Step counts around the 16-step blocks and the two steps of a Philox block; the spot far
    from 1 (no normalisation); jumps on about a quarter of the steps."""
    k = qk.make_contract(S0=250.0, v0=0.05, model=model, scheme=scheme, lambda_j=0.3 * n_steps if model else 0.0,
                         mu_j=-0.05, sigma_j=0.1, n_steps=n_steps, T=1.0, n_paths=70, seed=0xABCDEF0123, stream=3,
                         precision=qk.FP64, normalize=False)
    Sg, vg = qk.paths(k, 0, 70, handle)
    So, vo = oracle.paths(k, 0, 70)
    np.testing.assert_allclose(Sg, So, rtol=1e-12)
    np.testing.assert_allclose(vg, vo, rtol=2e-11, atol=4e-14)


@pytest.mark.parametrize("rho", [-0.9, 0.0, 0.9])
@pytest.mark.parametrize("v0,theta,kappa,sigma", [(0.01, 0.01, 0.5, 0.9), (0.04, 0.0, 0.0, 0.3), (0.09, 0.04, 2.0, 0.0)])
def test_fp64_qe_regimes_match_oracle(qk, handle, oracle, rho, v0, theta, kappa, sigma):
    """QE outside its quadratic regime: variance near zero (exponential regime), no mean
    reversion, and no vol-of-vol (the variance moves without noise)."""
    k = qk.make_contract(S0=100.0, v0=v0, theta=theta, kappa=kappa, sigma=sigma, rho=rho, scheme=qk.ANDERSEN_QE,
                         n_steps=64, T=2.0, n_paths=300, seed=77, precision=qk.FP64)
    Sg, vg = qk.paths(k, 0, 300, handle)
    So, vo = oracle.paths(k, 0, 300)
    np.testing.assert_allclose(Sg, So, rtol=1e-10)
    np.testing.assert_allclose(vg, vo, rtol=1e-8, atol=1e-13)


def test_fp64_spot_out_of_range_stays_ordered(qk, handle):
    """A variance so large that the spot underflows: prices stay finite and a put is worth its
    discounted strike."""
    k = qk.make_contract(v0=400.0, theta=400.0, kappa=1.0, sigma=0.5, rho=0.0, T=10.0, n_steps=20, n_paths=1000,
                         precision=qk.FP64, payoffs=[qk.payoff(qk.EUROPEAN, qk.PUT, 100.0), qk.payoff(qk.ASIAN, qk.CALL, 100.0)])
    legs = qk.price_plain(k, None, handle)["legs"]
    assert legs[0]["price"] == pytest.approx(100.0 * np.exp(-0.3), rel=1e-3)
    assert np.isfinite(legs[1]["price"])
