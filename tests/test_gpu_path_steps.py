"""GPU: the path loop's step code at the sizes where it can go wrong, against the oracle on
the same Philox draws.

Tolerances.  FP64: a step on the logarithm of the spot rounds a handful of times at a few
units in the last place (2^-52) of terms below 0.1, so 101 steps stay within 1e-13 of the
oracle; 1e-12 is asserted, as for the other FP64 path checks.  Next to zero variance QE's
(b + Z)^2 loses relative accuracy where b + Z cancels (b >= 0.7, so at most about 1e-12 of
a variance that small moves the spot by far less); 1e-10 on the spot there.
"""
import math

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


@pytest.mark.parametrize("model", [0, 1])
def test_qe_with_a_reachable_clamp(qk, handle, oracle, model):
    """Steps of five years with rho = 0.9: A a can pass 1/2, so min(A, 1/(2a) - eps) matters and
    no step may take the clamp-free form.  FP64 paths against the oracle; FP32 with one and two
    paths per lane simulates the same paths (prices to the rounding of the moment merge)."""
    base = dict(model=model, scheme=qk.ANDERSEN_QE, v0=0.3, theta=0.3, kappa=0.1, sigma=0.5, rho=0.9, T=10.0, n_steps=2,
                lambda_j=0.1 if model else 0.0, mu_j=-0.05, sigma_j=0.1, seed=9)
    k = qk.make_contract(n_paths=500, precision=qk.FP64, **base)
    Sg, _ = qk.paths(k, 0, 500, handle)
    So, _ = oracle.paths(k, 0, 500)
    np.testing.assert_allclose(Sg, So, rtol=1e-10)
    c = qk.make_contract(n_paths=20_001, precision=qk.FP32, payoffs=[qk.payoff(qk.EUROPEAN, qk.PUT, 100.0)], **base)
    out = []
    try:
        for lanes in (1, 2):
            handle.tune_set(qk.FP32, model, qk.ANDERSEN_QE, 24, False, lanes)
            out.append(qk.price_batch([c], None, handle)[0]["legs"][0]["price"])
    finally:
        handle.tune_reset()
    assert out[0] == pytest.approx(out[1], rel=1e-12)


@pytest.mark.parametrize("n_paths,n_steps", [(1, 1), (31, 63), (33, 64), (65, 65), (129, 130), (1000, 257)])
@pytest.mark.parametrize("model,scheme", [(0, 0), (1, 0), (1, 2)])
def test_generator_rows_at_warp_and_block_edges(qk, handle, oracle, model, scheme, n_paths, n_steps):
    """Path counts around a warp's 32 lanes (one or two paths each) and step counts around the
    64 steps a warp's generator rows cover: FP64 prices against the oracle's (1e-9, as the other
    price checks), FP32 with one and two paths per lane alike (to the rounding of the merge)."""
    base = dict(model=model, scheme=scheme, lambda_j=2.0 if model else 0.0, mu_j=-0.05, sigma_j=0.1, n_paths=n_paths,
                n_steps=n_steps, seed=(5 << 32) + 7, stream=2 ** 32 - 1,
                payoffs=[qk.payoff(qk.ASIAN, qk.CALL, 90.0), qk.payoff(qk.LOOKBACK_FLOATING, qk.PUT, 100.0)])
    k = qk.make_contract(precision=qk.FP64, **base)
    for got, want in zip(qk.price_batch([k], None, handle)[0]["legs"], oracle.price(k)["legs"]):
        assert got["price"] == pytest.approx(want["price"], rel=1e-9, abs=1e-12)
    c = qk.make_contract(precision=qk.FP32, **base)
    out = []
    try:
        for lanes in (1, 2):
            handle.tune_set(qk.FP32, model, scheme, 24, False, lanes)
            out.append([leg["price"] for leg in qk.price_batch([c], None, handle)[0]["legs"]])
    finally:
        handle.tune_reset()
    assert out[0] == pytest.approx(out[1], rel=1e-12, abs=1e-15)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n_paths", [33, 4096, 150_000, 151_553, 400_000])
def test_single_wave_launches_keep_the_bits(qk, handle, precision, n_paths):
    """Path counts on both sides of the line below which every tile gets a resident warp of its
    own (one-warp-per-scheduler blocks): the block size of persistent launches changes no bit."""
    c = qk.make_contract(scheme=qk.ANDERSEN_QE, n_paths=n_paths, n_steps=8, seed=3, precision=precision,
                         payoffs=[qk.payoff(qk.EUROPEAN, qk.CALL, 100.0), qk.payoff(qk.ASIAN, qk.CALL, 100.0)])
    out = []
    try:
        for block in (128, 256):
            handle.tune_set(precision, qk.HESTON, qk.ANDERSEN_QE, 24, False, 2 if precision else 1, block_size=block)
            out.append(qk.price_batch([c], None, handle)[0]["legs"])
    finally:
        handle.tune_reset()
    assert out[0] == out[1]


@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("params", [
    dict(sigma=0.3, rho=-0.7, T=0.1, n_steps=25),                         # term above 1, a few thousand floats
    dict(sigma=0.3, rho=0.6, T=0.1, n_steps=25),                          # term below 1
    dict(sigma=0.9, rho=-0.7, v0=0.01, theta=0.01, kappa=0.5, T=0.1, n_steps=25),  # many steps outside the plain regime
    dict(sigma=0.3, rho=0.0, T=0.1, n_steps=25),                          # term next to 1
    dict(sigma=0.3, rho=-0.7, theta=0.0, kappa=0.0, T=0.1, n_steps=25),   # no mean reversion
    dict(sigma=0.5, rho=-0.9, T=4.0, n_steps=9),                          # too many floats for a table
])
def test_term_table_keeps_the_bits(qk, handle, model, params):
    """A persistent launch of one FP32 QE contract in 512-thread blocks takes two SFU results per
    step from a table; blocks of 256 threads take none.  The same bits, also next to and outside
    the table's range."""
    c = qk.make_contract(model=model, scheme=qk.ANDERSEN_QE, lambda_j=0.4 if model else 0.0, mu_j=-0.05, sigma_j=0.1,
                         n_paths=1_000_003, seed=31, precision=qk.FP32,
                         payoffs=[qk.payoff(qk.EUROPEAN, qk.CALL, 100.0), qk.payoff(qk.ASIAN, qk.PUT, 100.0)], **params)
    out = []
    try:
        for block in (256, 512):
            handle.tune_set(qk.FP32, model, qk.ANDERSEN_QE, 24, False, 2, block_size=block)
            out.append(qk.price_batch([c], None, handle)[0]["legs"])
    finally:
        handle.tune_reset()
    assert out[0] == out[1]


@pytest.mark.parametrize("model", [0, 1])
def test_slab_term_table_keeps_the_bits(qk, handle, model):
    """American forward slabs of one FP32 QE contract: path counts below and above the line from
    which the slab kernel uses the table price like the FP64 engine (0.25 SE, as the other FP32
    American checks), and a contract equals itself priced in one call with another."""
    for n_paths in (100_001, 400_003):
        c = qk.make_contract(model=model, scheme=qk.ANDERSEN_QE, lambda_j=0.2 if model else 0.0, mu_j=-0.05, sigma_j=0.1,
                             n_paths=n_paths, n_steps=50, T=0.2, seed=8, precision=qk.FP32, lsm_basis=qk.LSM_POLY_SV,
                             lsm_dates=10, payoffs=[qk.payoff(qk.AMERICAN, qk.PUT, 100.0)])
        alone = qk.price_batch([c], None, handle)[0]["legs"][0]
        both = qk.price_batch([c, c], None, handle)
        assert both[0]["legs"][0] == both[1]["legs"][0] == alone
        if model == 0:  # Bates draws its jumps from other bits in FP64
            c64 = qk.make_contract(**{**dict(scheme=qk.ANDERSEN_QE, n_paths=n_paths, n_steps=50, T=0.2, seed=8,
                                             precision=qk.FP64, lsm_basis=qk.LSM_POLY_SV, lsm_dates=10),
                                      "payoffs": [qk.payoff(qk.AMERICAN, qk.PUT, 100.0)]})
            want = qk.price_plain(c64, None, handle)["legs"][0]
            assert abs(alone["price"] - want["price"]) < 0.25 * want["std_error"]


@pytest.mark.parametrize("n_contracts", [1, 5, 6, 30])
def test_results_on_both_sides_of_the_direct_write(qk, handle, n_contracts):
    """12 pricing tasks per contract: up to 64 tasks the merge writes the results to the host
    itself, beyond that they are copied; one-chunk and many-chunk tasks mixed.  A prepared set
    replayed (its queue cursors cleared by the run before) gives the one-shot call's results."""
    cs = [qk.make_contract(n_paths=3_000 + 40_000 * (i % 3), n_steps=6 + i % 5, seed=50 + i, scheme=i % 3,
                           precision=(qk.FP64, qk.FP32)[i % 2]) for i in range(n_contracts)]
    g = qk.make_greeks(qk.GREEK_ALL, bump_S_rel=0.01, bump_vol=0.02)
    want = qk.price_batch(cs, g, handle)
    for c, w in zip(cs, want):
        assert qk.price_batch([c], g, handle)[0]["legs"][0]["price"] == pytest.approx(w["legs"][0]["price"], rel=1e-13)
    prep = qk.PreparedBatch(cs, g, handle)
    for _ in range(3):
        prep.run()
        prep.run()
        assert [r["legs"] for r in prep.fetch()] == [r["legs"] for r in want]


@pytest.mark.parametrize("psi,v0,theta", [(1.5, 1e-3, 1e-3), (1.5 * (1 - 2.0**-19), 1e-3, 1e-3), (1.5 * (1 + 2.0**-19), 1e-3, 1e-3),
                                          (1e-6, 0.04, 0.04), (1e-6 * (1 + 2.0**-19), 0.04, 0.04), (0.5, 2e-6, 1e-7)])
@pytest.mark.parametrize("n_paths", [65, 1_000_003])
def test_qe_regime_bounds_keep_the_bits(qk, handle, n_paths, psi, v0, theta):
    """Paths that start with psi next to psi_c = 3/2, next to eps = 1e-6, and with a mean next to
    eps: two paths per lane (the regime from 2 / psi, with and without a term table) against the
    one-path step's comparisons.  The same paths bit for bit, so prices differ by the order of the
    FP64 merge alone."""
    kappa, dt = 2.0, 0.004
    e = math.exp(-kappa * dt)
    m = v0 * e + theta * (1 - e)
    s2 = v0 * e * (1 - e) / kappa + theta * (1 - e) ** 2 / (2 * kappa)  # over sigma^2
    c = qk.make_contract(scheme=qk.ANDERSEN_QE, v0=v0, theta=theta, kappa=kappa, sigma=math.sqrt(psi * m * m / s2), rho=-0.5,
                         n_steps=6, T=6 * dt, n_paths=n_paths, seed=77, precision=qk.FP32,
                         payoffs=[qk.payoff(qk.EUROPEAN, qk.CALL, 100.0), qk.payoff(qk.LOOKBACK_FLOATING, qk.PUT, 100.0)])
    out = []
    try:
        for lanes, block in ((1, 256), (2, 256), (2, 512)):
            handle.tune_set(qk.FP32, qk.HESTON, qk.ANDERSEN_QE, 24, False, lanes, block_size=block)
            out.append(qk.price_batch([c], None, handle)[0]["legs"])
    finally:
        handle.tune_reset()
    for legs in out[1:]:
        for a, b in zip(out[0], legs):
            assert a["prob_itm"] == b["prob_itm"]
            assert math.isclose(a["price"], b["price"], rel_tol=1e-11)
            assert math.isclose(a["std_error"], b["std_error"], rel_tol=1e-11)
