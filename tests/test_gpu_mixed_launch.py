"""Contracts of several kinds in one launch: averages beside Europeans whose
walks could be shared, in every order, on one stream. Every price equals the
contract's own call bit for bit."""
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

S = kx.S("X")
CALL, PUT = kx.european_call("X", 95.0, 1.0), kx.european_put("X", 100.0, 1.0)
ASIAN = kx.scale((kx.average(S) - 100.0).clip(0.0), kx.one()) @ kx.at(1.0)
LOOKBACK = kx.scale((kx.running_max(S) - 100.0).clip(0.0), kx.one()) @ kx.at(1.0)
MODELS = {
    "gbm": kx.GBM(s0=100.0, sigma=0.3, r=0.04, asset="X"),
    "heston": kx.heston(100.0, 0.04, 1.5, 0.04, 0.5, -0.7, 0.03, asset="X"),
}


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("model", sorted(MODELS))
def test_averages_beside_europeans(model, prec):
    m = MODELS[model]
    for cs in ([CALL, PUT, ASIAN], [ASIAN, CALL, PUT, CALL], [CALL, CALL, LOOKBACK], [ASIAN, CALL, PUT, LOOKBACK, PUT, PUT]):
        for n in (33, 2050):
            # larger paths of another stream first: what they leave in the launch's memory must not be read
            kx.price_portfolio(cs, [m] * len(cs), [4 * n] * len(cs), 99, steps_per_year=63, precision=prec)
            got = kx.price_portfolio(cs, [m] * len(cs), [n] * len(cs), 7, steps_per_year=63, precision=prec)
            for c, r in zip(cs, got):
                one = c.price(m, n_paths=n, seed=7, steps_per_year=63, precision=prec)
                assert (r.price, r.std_error) == (one.price, one.std_error)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_pairs_and_control_of_an_average_without_volatility(prec):
    """sigma = 0: the control and its mirror walk alike, and price - (control - Black-Scholes) is the payoff
    of the one path there is."""
    m = kx.GBM(s0=100.0, sigma=0.0, r=0.04, asset="X")
    kx.price_portfolio([ASIAN] * 4, [MODELS["gbm"]] * 4, [4000] * 4, 3, steps_per_year=50, precision=prec)
    plain = ASIAN.price(m, n_paths=2000, steps_per_year=50, precision=prec)
    both = ASIAN.price(m, n_paths=2000, steps_per_year=50, precision=prec, antithetic=True, control_variate=True)
    # the control's payoff is the Black-Scholes value but for the rounding of 50 steps
    tol = 100.0 * 50 * (2.0 ** -24 if prec == "fp32" else 2.0 ** -53) * 4
    assert abs(both.price - plain.price) <= tol
