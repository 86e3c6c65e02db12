"""GPU: American requests served while other lanes are busy get the price they get alone."""
import pytest

pytestmark = pytest.mark.gpu


def test_american_requests_in_a_burst_equal_alone(qk, handle):
    """The descriptors and centring constants of a wave's American jobs must have reached the
    device before its kernels read them, however busy the copy engine and the other lanes are:
    every result of repeated bursts equals the contract priced alone, bit for bit (the sweep's
    sums do not depend on what else runs)."""
    from quantkos_b200 import workloads as W
    _, contracts = W.serving_stream(60, seed=29)
    contracts = [c for c in contracts if c.payoffs[0].type == qk.AMERICAN][:14]
    for c in contracts:
        c.n_paths = min(c.n_paths, 600_000)
    want = [qk.price_batch([c], None, handle)[0]["legs"][0] for c in contracts]
    with qk.Server(handle, 8192) as srv:
        for _ in range(12):
            tickets = [srv.submit(c) for c in contracts]
            for t, w in zip(tickets, want):
                got = None
                while got is None:
                    got = srv.poll(t, 1000)
                assert got["legs"][0] == w
