"""Averages that walk on one draw (k_sync_scen: five or more FP32 GBM contracts
on the same paths, the same window and date) have each contract's own price bit
for bit: full and short last groups of seven, windows and dates that begin and
end inside a Philox block, grids around the 32 blocks whose words a warp keeps,
path counts around a warp, a spot so low that its exponential is subnormal."""
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

S = kx.S("X")
N = 35_000  # with five contracts and more: above the size from which one draw serves a group


def _asian(a, b, t):
    return kx.scale((kx.average_over(S, a, b) - 100.0).clip(0.0), kx.one()) @ kx.at(t)


def _models(k):
    return [kx.GBM(s0=100.0 + (i % 3), sigma=0.2 + 0.01 * i, r=0.03 + 0.001 * (i % 2), asset="X") for i in range(k)]


def _check(entries, spy):
    cs, ms, ns, seeds = zip(*entries)
    got = kx.price_portfolio(list(cs), list(ms), list(ns), list(seeds), steps_per_year=spy)
    assert kx.last_launch_stats()["path_kernel"] == 4
    for (c, m, n, seed), g in zip(entries, got):
        a = c.price(m, n_paths=n, seed=seed, steps_per_year=spy)
        assert (a.price, a.std_error) == (g.price, g.std_error)


@pytest.mark.parametrize("window", [(0.0, 1.0, 1.0), (0.26, 0.74, 1.0), (0.5, 1.0, 1.0), (0.0, 0.5, 0.8)])
@pytest.mark.parametrize("spy", [3, 63, 128, 131])
def test_windows_and_grids(window, spy):
    c = _asian(*window)
    _check([(c, m, N, 5) for m in _models(7)], spy)


@pytest.mark.parametrize("k", [5, 7, 8, 15])
@pytest.mark.parametrize("n", [N, N + 1, N + 31])
def test_groups_and_path_counts(k, n):
    c = kx.scale((kx.average(S) - 100.0).clip(0.0), kx.one()) @ kx.at(1.0)
    _check([(c, m, n, 9) for m in _models(k)], 50)


def test_subnormal_spot_in_a_group():
    c = kx.scale(kx.average(S), kx.one()) @ kx.at(1.0)
    low = kx.GBM(s0=100.0, sigma=0.3, r=0.0, q=90.0, asset="X")
    _check([(c, m, N, 3) for m in _models(6) + [low]], 50)


def test_strikes_and_payoffs_differ():
    cs = [kx.scale((kx.average(S) - k).clip(0.0), kx.one()) @ kx.at(1.0) for k in (90.0, 100.0, 110.0)]
    cs += [kx.scale((kx.S("X") - kx.average(S)).clip(0.0), kx.one()) @ kx.at(1.0)] * 3
    _check([(c, m, N, 4) for c, m in zip(cs, _models(6))], 52)
