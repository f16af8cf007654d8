"""k_tangent_walk against the general forward-mode kernel where the barrier's
window opens after t = 0 (inside a Philox block, at its edge, after the flow's
block begins) and where the flow under the barrier is a constant; the bound is
that of the other comparisons of the two kernels."""
import pytest
import test_gpu_tangent_walk as walk

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

S = kx.S("X")


def _late(t, cond=S >= 125.0):
    return kx.scale((S - 100.0).clip(0.0), kx.one()).when(kx.at(1.0)).until(cond).when(kx.at(t))


CONTRACTS = {
    "call_from_an_edge": lambda: _late(0.25),
    "call_from_inside": lambda: _late(21 / 64),
    "call_at_the_end": lambda: _late(61 / 64),
    "put_below": lambda: kx.scale((105.0 - S).clip(0.0), kx.one()).when(kx.at(1.0)).until(S < 85.0).when(kx.at(39 / 64)),
    "bond": lambda: kx.until(S >= 130.0, kx.zero_coupon_bond("USD", 1.0)),
    "late_bond": lambda: kx.zero_coupon_bond("USD", 1.0).until(S <= 90.0).when(kx.at(26 / 64)),
}


@pytest.mark.parametrize("name", sorted(CONTRACTS))
def test_matches_the_general_tangent_kernel(monkeypatch, name):
    c = CONTRACTS[name]()  # dates in 64ths: the grids are even
    for n, spy in ((1, 64), (129, 64), (1000, 128), (5000, 256), (300, 1024)):
        a = c.adjoint(walk.GBM, n_paths=n, seed=3, steps_per_year=spy)
        assert kx.last_launch_stats()["kernel"] == "k_tangent_walk", spy
        monkeypatch.setenv("KX_ADJOINT_KERNEL", "tangent")
        b = c.adjoint(walk.GBM, n_paths=n, seed=3, steps_per_year=spy)
        assert kx.last_launch_stats()["kernel"] == "k_tangent_gbm"
        monkeypatch.delenv("KX_ADJOINT_KERNEL")
        walk._close(a, b, n, 3 * spy)
