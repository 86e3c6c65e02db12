"""GPU: the FP64 pricing kernels' steps on the logarithm of the spot.

A call struck at 1e-4 of the spot pays the terminal spot (or the average) less the strike, so
the per-path payoffs show the pricing kernels' paths; they are compared with the oracle's on
the same draws.  Tolerances as for the paths: a step rounds a handful of terms below 0.1 at a few
units in the last place (2^-52), so 101 steps stay within 1e-13; 1e-12 is asserted, 1e-10
next to zero variance, where QE's (b + Z)^2 cancels, and where steps span years.
"""
import ctypes as C
import json
import math

import numpy as np
import pytest

from tests.helpers import GOLDEN

pytestmark = pytest.mark.gpu


def _check(qk, handle, oracle, rtol, types, **kw):
    """Per-path call payoffs struck at 1e-4 of the spot against the oracle's paths."""
    K = 1e-4 * kw.get("S0", 100.0)
    for t in types:
        k = qk.make_contract(precision=qk.FP64, payoffs=[qk.payoff(t, qk.CALL, K)], **kw)
        pay = np.empty(k.n_paths)
        assert qk.lib.lib().qk_payoffs_range(handle.ptr, C.byref(k), 0, k.n_paths, pay.ctypes.data_as(C.POINTER(C.c_double))) == 0
        S = oracle.paths(k, 0, k.n_paths)[0]
        S = S.mean(axis=1) if t == qk.ASIAN else S[:, -1]
        np.testing.assert_allclose(pay * k.S0 if k.normalize else pay, np.maximum(S - K, 0.0), rtol=rtol)


@pytest.mark.parametrize("n_steps", [1, 2, 15, 16, 17, 101])
@pytest.mark.parametrize("model,scheme", [(m, s) for m in (0, 1) for s in (0, 1, 2)])
def test_spots_at_block_edges_match_oracle(qk, handle, oracle, model, scheme, n_steps):
    _check(qk, handle, oracle, 1e-12, [qk.EUROPEAN], S0=250.0, v0=0.05, model=model, scheme=scheme,
           lambda_j=0.3 * n_steps if model else 0.0, mu_j=-0.05, sigma_j=0.1, n_steps=n_steps, T=1.0, n_paths=70,
           seed=0xABCDEF0123, stream=3, normalize=False)


@pytest.mark.parametrize("rho", [-0.9, 0.0, 0.9])
@pytest.mark.parametrize("v0,theta,kappa,sigma", [(0.01, 0.01, 0.5, 0.9), (0.04, 0.0, 0.0, 0.3), (0.09, 0.04, 2.0, 0.0)])
def test_qe_regimes_match_oracle(qk, handle, oracle, rho, v0, theta, kappa, sigma):
    _check(qk, handle, oracle, 1e-10, [qk.EUROPEAN], v0=v0, theta=theta, kappa=kappa, sigma=sigma, rho=rho,
           scheme=qk.ANDERSEN_QE, n_steps=64, T=2.0, n_paths=300, seed=77)


@pytest.mark.parametrize("dt", [1.0 / 252, 0.06, 0.15, 0.25, 0.5, 1.0, 2.0, 4.0])
@pytest.mark.parametrize("rho", [-0.9, 0.5, 0.9])
def test_qe_product_at_every_fold_interval(qk, handle, oracle, rho, dt):
    """Variances that stay in the quadratic regime and factors 1 - 2 A a from next to 1 down to the
    clamp: the product is folded every 16, 8, 4 or 2 steps, and at the last no step multiplies.
    Where most spots end below the strike, the average still reads them."""
    _check(qk, handle, oracle, 1e-10, [qk.EUROPEAN, qk.ASIAN], v0=0.8, theta=0.8, kappa=2.0, sigma=0.9, rho=rho,
           scheme=qk.ANDERSEN_QE, n_steps=37, T=37 * dt, n_paths=300, seed=78)


@pytest.mark.parametrize("leg", ["asian", "european"])
def test_qe_prices_against_long_double(qk, handle, leg):
    """Ten contracts of 100,003 paths by 126 steps, priced in long double on the same draws from
    the same (rounded) step constants.  The textbook's formulas in FP64 are off by 2e-16 to 4e-16
    (root mean square of the relative errors), a product of rho / sigma rounded apart from the
    one it cancels with by 4e-15; 1e-15 is asserted."""
    err = []
    for r in json.loads((GOLDEN / "heston_qe_long_double.json").read_text()):
        if r["leg"] != leg:
            continue
        k = qk.make_contract(S0=100.0, v0=r["v0"], r=0.03, q=0.0, scheme=qk.ANDERSEN_QE, kappa=2.0, theta=0.04, sigma=r["sigma"],
                             rho=r["rho"], T=0.5, n_steps=126, n_paths=100_003, seed=r["seed"], precision=qk.FP64,
                             payoffs=[qk.payoff(qk.ASIAN if leg == "asian" else qk.EUROPEAN, qk.CALL, r["strike"])])
        got = np.longdouble(qk.price_plain(k, None, handle)["legs"][0]["price"])
        err.append(float(got / np.longdouble(r["price"]) - 1))
    assert len(err) == 10
    assert math.sqrt(np.mean(np.square(err))) < 1e-15, err


@pytest.mark.parametrize("antithetic", [False, True])
@pytest.mark.parametrize("model,scheme", [(0, 0), (0, 1), (0, 2), (1, 2)])
@pytest.mark.parametrize("n_steps", [1, 3, 16, 17])
def test_lookback_of_a_path_ending_at_its_extreme_pays_nothing(qk, handle, oracle, n_steps, model, scheme, antithetic):
    """Floating lookbacks on a spot of 20,000 without normalisation: a unit in the last place of
    the spot passes the in-the-money threshold of 1e-12, so the terminal spot and the running
    extreme it reaches have to be the same number.  The oracle takes both from one value."""
    k = qk.make_contract(S0=20_000.0, v0=0.04, model=model, scheme=scheme, lambda_j=0.2 if model else 0.0, mu_j=-0.05,
                         sigma_j=0.1, n_steps=n_steps, T=0.1, n_paths=4000, seed=21, precision=qk.FP64, normalize=False,
                         antithetic=antithetic, payoffs=[qk.payoff(qk.LOOKBACK_FLOATING, qk.CALL, 20_000.0),
                                                         qk.payoff(qk.LOOKBACK_FLOATING, qk.PUT, 20_000.0)])
    for got, want in zip(qk.price_batch([k], None, handle)[0]["legs"], oracle.price(k)["legs"]):
        assert got["prob_itm"] == pytest.approx(want["prob_itm"], abs=1e-9)
        assert got["price"] == pytest.approx(want["price"], rel=1e-9)
