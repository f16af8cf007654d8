"""k_knock (one-flow knock-outs and knock-ins, the barriers looked at once per
segment of Philox blocks) values every path as the general kernel does, bit for
bit: path counts around a warp, a group of warps and a block's list, grids that
end inside a block and inside a segment, up, down and double barriers, strict
and inclusive, a path knocked out or in at t = 0, the longest grid served and
one beyond it, a grid whose steps are not equal in FP32; knock-ins that miss
the pattern (a flow due before the last step) still price."""
import numpy as np
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

S = kx.S("X")

CONTRACTS = {
    "up_out": lambda: kx.up_and_out_call("X", 100.0, 120.0, 1.0),
    "up_out_strict": lambda: kx.until(S > 120.0, kx.european_call("X", 100.0, 1.0)),
    "down_out_put": lambda: kx.until(S < 85.0, kx.european_put("X", 105.0, 1.0)),
    "double": lambda: kx.until(S >= 125.0, kx.until(S <= 85.0, kx.european_call("X", 100.0, 1.0))),
    "two_up": lambda: kx.until(S >= 125.0, kx.until(S > 118.0, kx.give(kx.european_call("X", 100.0, 1.0)))),
    "rebate": lambda: kx.until(S <= 80.0, kx.scale(7.5, kx.one()) @ kx.at(1.0)) + kx.one(),
    "knocked_at_zero": lambda: kx.until(S <= 200.0, kx.european_call("X", 100.0, 1.0)),
    "up_in": lambda: kx.when(S >= 115.0, kx.european_call("X", 100.0, 1.0)),
    "down_in_strict": lambda: kx.anytime(S < 88.0, kx.give(kx.european_put("X", 100.0, 1.0))),
    "in_at_zero": lambda: kx.when(S <= 100.0, kx.european_put("X", 100.0, 1.0)),
    "in_pays_one": lambda: kx.when(S > 110.0, kx.zero_coupon_bond("USD", 1.0)),
    "in_early_flow": lambda: kx.when(S >= 110.0, kx.european_call("X", 100.0, 0.5) + kx.european_call("X", 90.0, 1.0)),
}


def _both(monkeypatch, c, m, n, spy, prec, seed=5):
    r1, p1 = c.price(m, n_paths=n, seed=seed, steps_per_year=spy, precision=prec, per_path=True)
    assert kx.last_launch_stats()["path_kernel"] in (2, 3)
    monkeypatch.setenv("KX_PATH_KERNEL", "general")
    r2, p2 = c.price(m, n_paths=n, seed=seed, steps_per_year=spy, precision=prec, per_path=True)
    monkeypatch.delenv("KX_PATH_KERNEL")
    assert np.array_equal(np.asarray(p1), np.asarray(p2))
    assert r1.price == r2.price and r1.std_error == r2.std_error


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("name", sorted(CONTRACTS))
def test_equals_the_general_kernel(monkeypatch, name, prec):
    m = kx.GBM(s0=100.0, sigma=0.3, r=0.04, asset="X")
    for n, spy in ((1, 2), (31, 3), (33, 4), (1000, 31), (257, 64), (4097, 66), (65, 255), (40, 1024), (40, 1025)):
        _both(monkeypatch, CONTRACTS[name](), m, n, spy, prec)


def test_lists_of_many_blocks(monkeypatch):
    """Enough paths that a block's lists are full and its tail items short."""
    m = kx.GBM(s0=100.0, sigma=0.4, r=0.02, asset="X")
    for c in (CONTRACTS["up_out"](), CONTRACTS["double"](), CONTRACTS["up_in"]()):
        _both(monkeypatch, c, m, 1_500_001, 30, "fp32")
    _both(monkeypatch, CONTRACTS["up_out"](), m, 300_001, 30, "fp64")


def _steps_differ(m, maturity, spy):
    n = int(np.ceil(maturity * spy))
    dt = np.diff(np.array([maturity * k / n for k in range(n + 1)]))
    c0 = ((m.r - 0.5 * m.sigma * m.sigma) * dt).astype(np.float32)
    c1 = (m.sigma * np.sqrt(dt)).astype(np.float32)
    return len(np.unique(c0)) > 1 or len(np.unique(c1)) > 1


def test_unequal_steps_and_a_book_that_meets_them(monkeypatch):
    """A maturity whose FP32 steps are equal under one volatility and not under
    another: the price equals the general kernel's under both, and a book
    created under the first prices the second after set_models."""
    c = kx.up_and_out_call("X", 100.0, 130.0, 1.3)
    even = kx.GBM(s0=100.0, sigma=0.3, r=0.03, asset="X")
    odd = kx.GBM(s0=100.0, sigma=0.460281, r=0.03, asset="X")
    assert not _steps_differ(even, 1.3, 252) and _steps_differ(odd, 1.3, 252)
    for m in (even, odd):
        _both(monkeypatch, c, m, 3000, 252, "fp32")
    d = kx.when(S <= 85.0, kx.european_put("X", 100.0, 1.3))
    for first in (even, odd):
        book = kx.Book([c, c, d], [first] * 3, [3000, 70_000, 5000], [5, 6, 7], steps_per_year=252)
        assert book.info()["n_groups"] == 2
        for m in (even, odd, even):
            book.set_models([m] * 3)
            for r, k, n, s in zip(book.price(), (c, c, d), (3000, 70_000, 5000), (5, 6, 7)):
                assert r.price == k.price(m, n_paths=n, seed=s, steps_per_year=252).price
        book.close()
