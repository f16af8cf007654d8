"""k_flows_walk (a book's flows on one simulation, the threads of a block in
step): each contract's statistics equal its own price on the same grid exactly
where the grids agree (the FP32 amounts are discounted with integer multiplies
that must give the FP64 product's bits), for path counts around a block, flows
inside a Philox block, both models and schemes, and on either side of the
longest grid whose tables fit shared memory."""
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

MODELS = {
    "gbm": kx.GBM(s0=100.0, sigma=0.3, r=0.04, asset="X"),
    "heston": kx.heston(100.0, 0.04, 1.5, 0.05, 0.6, -0.7, 0.03, asset="X"),
    "heston_ft": kx.heston(100.0, 0.04, 1.5, 0.05, 0.6, -0.7, -0.02, asset="X", scheme="full_truncation"),
}


def _book(t):
    return [kx.european_call("X", 100.0, t), kx.european_put("X", 90.0, t), kx.give(kx.european_call("X", 120.0, t)),
            kx.european_call("X", 400.0, t), kx.european_put("X", 99.99, t), kx.zero_coupon_bond("USD", t),
            kx.scale(2.0 * kx.S("X") - 150.0, kx.one()) @ kx.at(t)]


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("model", sorted(MODELS))
def test_same_maturity_equals_own_price(model, prec):
    m = MODELS[model]
    for n, spy, t in ((1, 1, 1.0), (255, 3, 1.0), (257, 9, 0.9), (1000, 63, 1.3), (40, 2000, 1.0)):
        book = _book(t)
        for c, r in zip(book, kx.price_batch(book, m, n_paths=n, seed=11, steps_per_year=spy, precision=prec)):
            one = c.price(m, n_paths=n, seed=11, steps_per_year=spy, precision=prec)
            assert r.price == one.price and r.std_error == one.std_error, (c, n, spy)


@pytest.mark.parametrize("model", ["gbm", "heston"])
def test_flows_inside_blocks_and_long_grids(model):
    """Contracts of several dates on the merged grid: a book split in two gives the whole book's values where
    the grid is the same, and a grid whose tables do not fit a block (8,000 Heston steps) prices as one that does."""
    m = MODELS[model]
    dates = [0.1, 0.25, 0.5, 0.51, 1.0]
    book = [kx.european_call("X", 100.0, t) for t in dates] + [kx.straddle("X", 95.0, 1.0)]
    for spy in (10, 100, 8000):
        n = 300 if spy < 8000 else 20
        whole = kx.price_batch(book, m, n_paths=n, seed=4, steps_per_year=spy, precision="fp32")
        for i in range(len(dates)):  # the dates stay on the grid as bonds
            part = [book[i]] + [kx.zero_coupon_bond("USD", t) for t in dates]
            assert kx.price_batch(part, m, n_paths=n, seed=4, steps_per_year=spy, precision="fp32")[0].price == whole[i].price
        own = book[5].price(m, n_paths=n, seed=4, steps_per_year=spy, precision="fp32")
        assert abs(whole[5].price - own.price) < 4 * (own.std_error + whole[5].std_error) + 1e-6
