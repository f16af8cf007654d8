"""k_sync (static schedules without barriers, the lanes of a warp in step)
values every path as the general kernel does, bit for bit: path counts around
a warp, grids around its Philox blocks (4 GBM or 2 Heston steps) and around the
32 blocks whose shared words a warp keeps, events and accumulator windows that
begin and end inside a block, a spot so low that its exponential is subnormal."""
import numpy as np
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

S = kx.S("X")


def _asian(a, b, t=1.0):
    return kx.scale((kx.average_over(S, a, b) - 100.0).clip(0.0), kx.one()) @ kx.at(t)


CONTRACTS = {
    "call": lambda: kx.european_call("X", 100.0, 1.0),
    "strip": lambda: kx.european_call("X", 100.0, 0.3) + kx.european_put("X", 105.0, 0.61) + kx.european_call("X", 95.0, 1.0),
    "asian": lambda: kx.scale((kx.average(S) - 100.0).clip(0.0), kx.one()) @ kx.at(1.0),
    "asian_window": lambda: _asian(0.26, 0.74),
    "asian_early": lambda: _asian(0.0, 0.5, 0.8) + kx.european_call("X", 100.0, 0.9),
    "lookback": lambda: kx.scale((kx.running_max(S) - 100.0).clip(0.0), kx.one()) @ kx.at(1.0),
    "lookback_put": lambda: kx.scale((105.0 - kx.running_min(S)).clip(0.0), kx.one()) @ kx.at(0.8),
    "bond": lambda: kx.zero_coupon_bond("USD", 0.7),
}
GBM = kx.GBM(s0=100.0, sigma=0.3, r=0.04, asset="X")
HESTON = kx.heston(100.0, 0.04, 1.5, 0.04, 0.5, -0.7, 0.03, asset="X")


def _both(monkeypatch, c, m, n, spy, prec, seed=5):
    r1, p1 = c.price(m, n_paths=n, seed=seed, steps_per_year=spy, precision=prec, per_path=True)
    assert kx.last_launch_stats()["path_kernel"] in (3, 4)
    monkeypatch.setenv("KX_PATH_KERNEL", "general")
    r2, p2 = c.price(m, n_paths=n, seed=seed, steps_per_year=spy, precision=prec, per_path=True)
    assert kx.last_launch_stats()["path_kernel"] == 1
    monkeypatch.delenv("KX_PATH_KERNEL")
    assert np.array_equal(np.asarray(p1), np.asarray(p2))
    assert r1.price == r2.price and r1.std_error == r2.std_error
    return np.asarray(p1)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("name", sorted(CONTRACTS))
def test_equals_the_general_kernel(monkeypatch, name, prec):
    for n, spy in ((1, 3), (31, 4), (33, 5), (1000, 63), (257, 128), (257, 129), (65, 515)):
        _both(monkeypatch, CONTRACTS[name](), GBM, n, spy, prec)
    for n, spy in ((33, 2), (1000, 63), (65, 131)):
        _both(monkeypatch, CONTRACTS[name](), HESTON, n, spy, prec)


def test_subnormal_spots(monkeypatch):
    """A drift of -90 a year takes the spot through the subnormal range of e^y."""
    m = kx.GBM(s0=100.0, sigma=0.3, r=0.0, q=90.0, asset="X")
    c = kx.scale(kx.running_min(S), kx.one()) @ kx.at(1.0)
    assert _both(monkeypatch, c, m, 500, 50, "fp32").max() < 1e-30
    _both(monkeypatch, CONTRACTS["asian"](), m, 500, 50, "fp32")


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("n", [1, 33, 2050])
def test_jobs_that_share_walks_and_normals(prec, n):
    """A launch of several contracts on one stream: Europeans under models that
    differ in the spot alone share their walks, and the FP64 walks of one stream
    read one table of normals. Every price equals the contract's own call."""
    g = [kx.GBM(s0=s, sigma=v, r=0.04, asset="X") for s, v in ((100.0, 0.3), (101.0, 0.3), (99.0, 0.3), (100.0, 0.2))]
    h = [kx.heston(s, v0, 1.5, 0.04, 0.5, -0.7, 0.03, asset="X") for s, v0 in ((100.0, 0.04), (90.0, 0.04), (100.0, 0.05))]
    call, put, asian = CONTRACTS["call"](), kx.european_put("X", 95.0, 1.0), CONTRACTS["asian"]()
    early = kx.european_call("X", 100.0, 0.6)
    books = [([call] * 4, g), ([call, put, call], g[:3]), ([call, early, call], [g[0]] * 3), ([asian] * 3, [g[0], g[1], g[3]]),
             ([call] * 3, h), ([call, put], [h[0], h[0]])]
    for cs, ms in books:
        for seeds in (7, list(range(7, 7 + len(cs)))):
            got = kx.price_portfolio(cs, ms, [n] * len(cs), seeds, steps_per_year=63, precision=prec)
            for i, (c, m, r) in enumerate(zip(cs, ms, got)):
                one = c.price(m, n_paths=n, seed=7 if seeds == 7 else seeds[i], steps_per_year=63, precision=prec)
                assert r.price == one.price and r.std_error == one.std_error
    uneven = kx.price_portfolio([call, call], g[:2], [n, n + 5], 7, steps_per_year=63, precision=prec)
    for m, k, r in zip(g, (n, n + 5), uneven):
        assert r.price == call.price(m, n_paths=k, seed=7, steps_per_year=63, precision=prec).price
