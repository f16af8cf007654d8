"""steps_simulated counts the steps a launch walks, those behind a path's
knock-out up to its segment's end among them. Without volatility every path
meets the barrier at the same known step, so the count lies between that step
and the grid's end for each path."""
import math

import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("barrier", [100.5, 101.0, 102.0, 103.9])
def test_paths_knocked_out_inside_a_segment(prec, barrier):
    n, spy = 1000, 256
    hit = math.ceil(math.log(barrier / 100.0) / 0.04 * spy)
    m = kx.GBM(s0=100.0, sigma=0.0, r=0.04, asset="X")
    r = kx.up_and_out_call("X", 100.0, barrier, 1.0).price(m, n_paths=n, steps_per_year=spy, precision=prec)
    st = kx.last_launch_stats()
    assert st["kernel"] == "k_knock" and r.price == 0.0
    assert n * hit <= st["steps_simulated"] <= n * spy

    mm = kx.CorrelatedGbmN([("A", 100.0, 0.04, 0.0), ("B", 100.0, 0.04, 0.0)], [[1.0, 0.2], [0.2, 1.0]], rate=0.04)
    basket = (kx.S("A") + kx.S("B")) / 2.0
    c = kx.until(basket >= barrier, kx.scale((basket - 100.0).clip(0.0), kx.one()) @ kx.at(1.0))
    r = c.price(mm, n_paths=n, steps_per_year=spy, precision=prec)
    st = kx.last_launch_stats()
    assert st["kernel"] == "k_multi_knock" and r.price == 0.0
    assert n * hit <= st["steps_simulated"] <= n * spy


def test_paths_that_live_count_every_step():
    m = kx.GBM(s0=100.0, sigma=0.0, r=0.04, asset="X")
    kx.up_and_out_call("X", 100.0, 200.0, 1.0).price(m, n_paths=1000, steps_per_year=255)
    assert kx.last_launch_stats()["steps_simulated"] == 1000 * 255


def test_forward_sensitivities_walk_to_the_flow_once():
    m = kx.GBM(s0=100.0, sigma=0.3, r=0.04, asset="X")
    c = kx.scale((kx.average_over(kx.S("X"), 0.0, 0.5) - 100.0).clip(0.0), kx.one()) @ kx.at(0.75)
    c.adjoint(m, n_paths=1000, steps_per_year=64)
    st = kx.last_launch_stats()
    assert st["kernel"] == "k_tangent_walk" and st["steps_simulated"] == 1000 * 48
