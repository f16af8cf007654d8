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
