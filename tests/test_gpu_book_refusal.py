"""A book whose new models are refused keeps its market whole: neither the
tables nor the captured launches of the groups planned before the refusal
change, whichever kernel those groups would have moved to."""
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

S = kx.S("X")
# FP32 steps of 1.3 years at 252 a year are equal under the first volatility and not under the second:
# the knock-outs run on k_knock under one and on k_lean under the other
EVEN = kx.GBM(s0=100.0, sigma=0.3, r=0.03, asset="X")
ODD = kx.GBM(s0=100.0, sigma=0.460281, r=0.03, asset="X")
KO = kx.up_and_out_call("X", 100.0, 130.0, 1.3)
# price-triggered, flows at two dates: priced in log-space unless the spot is not positive, which changes its kernel
LATER = kx.when(S >= 110.0, kx.european_call("X", 100.0, 0.5) + kx.european_call("X", 90.0, 1.3))
REFUSED = kx.GBM(s0=0.0, sigma=0.3, r=0.03, asset="X")
N, SEED = (70_000, 3000, 5000), (5, 6, 7)


def _prices(m):
    return [c.price(m, n_paths=n, seed=s, steps_per_year=252).price for c, n, s in zip((KO, KO, LATER), N, SEED)]


@pytest.mark.parametrize("first,second", [(EVEN, ODD), (ODD, EVEN)], ids=["knock_to_lean", "lean_to_knock"])
def test_a_refused_market_changes_nothing(first, second):
    book = kx.Book([KO, KO, LATER], [first] * 3, list(N), list(SEED), steps_per_year=252)
    old = _prices(first)
    assert [r.price for r in book.price()] == old
    for _ in range(2):
        with pytest.raises(kx.KontractError) as e:
            book.set_models([second, second, REFUSED])
        assert "kernel family" in str(e.value)
        assert [r.price for r in book.price()] == old
    book.set_models([second] * 3)
    assert [r.price for r in book.price()] == _prices(second)
    book.set_models([first] * 3)
    assert [r.price for r in book.price()] == old
    book.close()
