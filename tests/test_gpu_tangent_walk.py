"""k_tangent_walk (FP32 GBM contracts of one flow on one average or under one
smoothed barrier, threads in step) against the general forward-mode kernel:
the same prices and payoffs bit for bit, and sensitivities that differ at most
by the rounding of a path's sums (steps * 2^-24 of the size of its terms, the
mean's plus a standard deviation). Path counts around a block, grids around a
Philox block of 4 steps, windows that begin and end inside one, a barrier that
arms late, a portfolio of uneven contracts."""
import math

import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

S = kx.S("X")


def _asian(a, b, t):
    return kx.scale((kx.average_over(S, a, b) - 100.0).clip(0.0), kx.one()) @ kx.at(t)


CONTRACTS = {
    "asian": lambda: kx.scale((kx.average(S) - 100.0).clip(0.0), kx.one()) @ kx.at(1.0),
    "asian_window": lambda: _asian(0.25, 0.75, 1.0),
    "asian_early": lambda: _asian(0.0, 0.5, 0.75),
    "floating": lambda: kx.scale((S - kx.average(S)).clip(0.0), kx.one()) @ kx.at(1.0),
    "up_and_out": lambda: kx.up_and_out_call("X", 100.0, 130.0, 1.0),
    "down_and_out": lambda: kx.scale((S - 100.0).clip(0.0), kx.one()).when(kx.at(1.0)).until(S < 85.0),
}
GBM = kx.GBM(s0=100.0, sigma=0.3, r=0.04, asset="X")
FIELDS = ("d_s0", "d_sigma", "d_r")


def _close(a, b, n, steps):
    assert a.price == b.price and a.price_se == b.price_se
    for f in FIELDS:
        x, y, se = getattr(a, f), getattr(b, f), getattr(b, f.replace("d_", "se_"))
        assert abs(x - y) <= steps * 2.0 ** -24 * (abs(y) + (se if math.isfinite(se) else 0.0) * math.sqrt(n)), (f, x, y)


@pytest.mark.parametrize("name", sorted(CONTRACTS))
def test_matches_the_general_tangent_kernel(monkeypatch, name):
    c = CONTRACTS[name]()
    for n, spy in ((1, 4), (127, 8), (129, 12), (1000, 64), (5000, 252), (300, 1200)):
        a = c.adjoint(GBM, n_paths=n, seed=3, steps_per_year=spy)
        monkeypatch.setenv("KX_ADJOINT_KERNEL", "tangent")
        b = c.adjoint(GBM, n_paths=n, seed=3, steps_per_year=spy)
        monkeypatch.delenv("KX_ADJOINT_KERNEL")
        _close(a, b, n, 3 * spy)


@pytest.mark.parametrize("kind", [("asian", "floating", "asian"), ("up_and_out", "down_and_out", "up_and_out")])
def test_portfolio(monkeypatch, kind):
    cs = [CONTRACTS[k]() for k in kind]
    ms = [GBM, kx.GBM(s0=95.0, sigma=0.2, r=0.01, asset="X"), kx.GBM(s0=110.0, sigma=0.25, r=0.03, asset="X")]
    ns = [130, 1, 777]
    pa, a = kx.price_portfolio(cs, ms, ns, [1, 2, 3], steps_per_year=100, greeks=True)
    monkeypatch.setenv("KX_ADJOINT_KERNEL", "tangent")
    pb, b = kx.price_portfolio(cs, ms, ns, [1, 2, 3], steps_per_year=100, greeks=True)
    for x, y, u, v, n in zip(pa, pb, a, b, ns):
        assert x.price == y.price
        _close(u, v, n, 300)
