"""GPU: the payoff percentiles are exact order statistics of the per-path payoffs."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FRACTIONS = [0.01, 0.05, 0.10, 0.20, 0.30, 0.40, 0.50, 0.60, 0.70, 0.80, 0.90, 0.95, 0.99]


@pytest.mark.parametrize("n_paths", [1, 2, 31, 2048, 2049, 100_003])
@pytest.mark.parametrize("opt_type,precision", [(0, 0), (1, 1), (8, 0), (6, 1)])
def test_percentiles_equal_the_sorted_payoffs(qk, handle, n_paths, opt_type, precision):
    """Sizes around the selection's blocks; payoffs with many ties (out-of-the-money zeros, a
    binary's two values) and without (lookback).  Equal bit for bit to sorting qk_payoffs_range."""
    cfg = qk.UInputs()
    for k, v in dict(v0=0.04, r=0.05, opt_type=opt_type, opt_right=1 if opt_type == 6 else 0, K=105.0, scheme=2, t_end=1.0,
                     inp_dt=1.0 / 20, n_paths=n_paths, seed=4242, precision=precision, engine=1 if precision else 0,
                     analyze_distribution=1, out_dir="", paths_file="").items():
        setattr(cfg, k, v)
    got = list(qk.MCDispatcher(cfg.validate(), handle).launch_montecarlo().OptionPrice.percentiles.values())
    k, _ = cfg.to_contract()
    pay = np.empty(n_paths)
    assert qk.lib.lib().qk_payoffs_range(handle.ptr, C.byref(k), 0, n_paths, pay.ctypes.data_as(C.POINTER(C.c_double))) == 0
    pay.sort()
    eff = math.exp(-0.05) * (1.0 if opt_type == 8 else 100.0)
    want = [pay[0] * eff] + [pay[int(n_paths * f)] * eff for f in FRACTIONS] + [pay[-1] * eff]
    assert got == want


@pytest.mark.parametrize("n_paths", [1, 32, 33, 64, 65, 2049, 100_003])
@pytest.mark.parametrize("opt_type,precision,engine", [(0, 0, 0), (1, 0, 1), (1, 1, 1), (6, 1, 1), (0, 1, 0)])
def test_price_beside_the_distribution_equals_the_price_alone(qk, handle, n_paths, opt_type, precision, engine):
    """One simulation serves both (tile records formed from the stored payoffs); (0, 1, 0) prices in
    FP64 and selects from FP32 payoffs, two simulations.  FP64 rounding of a step's few operations
    over 20 steps stays below 1e-12 of the price."""
    res = []
    for analyze in (0, 1):
        cfg = qk.UInputs()
        for k, v in dict(v0=0.04, r=0.05, opt_type=opt_type, opt_right=1 if opt_type == 6 else 0, K=100.0, scheme=2,
                         t_end=1.0, inp_dt=1.0 / 20, n_paths=n_paths, seed=99, precision=precision, engine=engine,
                         analyze_distribution=analyze, out_dir="", paths_file="").items():
            setattr(cfg, k, v)
        res.append(qk.MCDispatcher(cfg.validate(), handle).launch_montecarlo().OptionPrice)
    alone, both = res
    assert math.isclose(both.option_price, alone.option_price, rel_tol=1e-12, abs_tol=1e-300)
    assert math.isclose(both.standard_error, alone.standard_error, rel_tol=1e-12, abs_tol=1e-300)
    assert both.prob_itm == alone.prob_itm
