"""GPU: FP64 American prices and path dumps keep the values that the engine has given since its
FP64 paths step the spot with the CUDA library's functions.

golden/american_fp64.json holds such values (floats in hexadecimal, SHA-256 of the dumped
arrays).  The reference's mode solves unscaled normal equations, so other last bits in the
paths can flip exercise decisions and move a price by 1e-4 of itself; without a flip, what is
left is the order of FP64 sums over at most 300,001 cash flows, below 1e-12.
"""
import hashlib
import json

import numpy as np
import pytest

from tests.helpers import GOLDEN

pytestmark = pytest.mark.gpu

DATA = json.loads((GOLDEN / "american_fp64.json").read_text())


@pytest.mark.parametrize("case", DATA["american"], ids=lambda c: "-".join(str(v) for k, v in c.items() if k != "want"))
def test_american_results_keep_their_values(qk, handle, case):
    kw = {k: v for k, v in case.items() if k != "want"}
    c = qk.make_contract(S0=100.0, v0=0.045, sigma=0.3, rho=-0.7, T=0.4, lambda_j=0.2 if kw["model"] else 0.0, mu_j=-0.05,
                         sigma_j=0.1, seed=11, precision=qk.FP64, payoffs=[qk.payoff(qk.AMERICAN, qk.PUT, 101.0)], **kw)
    want = [float.fromhex(x) for x in case["want"]]
    for leg in (qk.price_plain(c, None, handle)["legs"][0], qk.price_batch([c], None, handle)[0]["legs"][0]):
        assert [leg["price"], leg["std_error"], leg["prob_itm"]] == pytest.approx(want, rel=1e-12)


@pytest.mark.parametrize("case", DATA["paths"], ids=lambda c: f"{c['model']}-{c['scheme']}-{c['params']['v0']}")
def test_path_dumps_keep_their_bits(qk, handle, case):
    c = qk.make_contract(model=case["model"], scheme=case["scheme"], lambda_j=5.0 if case["model"] else 0.0, mu_j=-0.05,
                         sigma_j=0.1, S0=250.0, T=1.0, n_steps=101, n_paths=1000, seed=5, precision=qk.FP64,
                         normalize=False, **case["params"])
    for got, want in zip(qk.paths(c, 3, 997, handle), (case["spot_sha256"], case["variance_sha256"])):
        assert hashlib.sha256(np.ascontiguousarray(got).tobytes()).hexdigest() == want
